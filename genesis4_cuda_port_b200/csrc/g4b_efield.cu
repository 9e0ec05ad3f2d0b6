// g4b_efield.cu -- short-range longitudinal space charge on the device.
//
// The reference keeps the space-charge solver on the host: with short-range
// space charge on, BeamSolverCUDA::advance calls EFieldSolver::shortRange for
// every slice on the host particle copies and uploads a per-particle field
// (getEField(ip) + slice loss) that the push reads in place of the slice loss
// (src/Core/BeamSolverCUDA.cpp:523-547, 184-195, 633-680).  Here the whole
// step stays on the device: a cluster of CTAs per slice builds the slice's azimuthal
// and longitudinal density modes on a radial grid, solves one tridiagonal
// system per mode and writes every particle's field into the beam's
// per-particle buffer, which the push then reads.
//
// Model (per slice, particles i = 1..N, current I):
//   density modulation at harmonic l of the reference wavelength, azimuthal
//   order m:  S_lm(r) = (1/N) sum_i delta(r - r_i) e^{-i(l theta_i + m phi_i)}
//   (radial cell average),
//   (1/r d/dr r d/dr - m^2/r^2 - kappa_l^2) u_lm = -S_lm,  kappa_l = l k_s / gamma_z,
//   u = 0 on the wall r = R, R = rmax * (largest particle radius about the
//   slice centroid),
//   E_z = sum_{l>=1} 2 Re[ i l k_s I Z0 / gamma_z^2 u_l e^{i l theta} ]
//   (the quasi-static field of a modulation moving with the beam), and the
//   push's loss term ez = E_z / (m_e c^2 / e) + slice loss.
// Discretisation: N radial cells of width dr = R/N, centres (j+1/2) dr,
// finite-volume fluxes through the cell faces, the wall half a cell beyond
// the last centre.  Mode sums are exact 2^-40 fixed-point integers (shared
// 64-bit atomics), so the result does not depend on particle order.

#include <algorithm>
#include <cmath>
#include <new>

#include "g4b_internal.cuh"

namespace g4b {
namespace {

constexpr int kScThreads = 256;
constexpr double kScFix = 1099511627776.0;  // 2^40
constexpr double kScUnfix = 1.0 / 1099511627776.0;
constexpr int64_t kScMaxSliceNp = int64_t(1) << 22;  // |mode sum| < 2^62
constexpr double kVacImp = 376.73031346177;   // Z0 [Ohm]
constexpr double kEev = 510998.95;            // m_e c^2 / e [V]

struct ScArgs {
  const double *x, *y, *theta;
  const int64_t* off;
  const double* current;  // [A] per slice
  const double* eloss;    // per-slice loss the push would otherwise use
  double* pez;            // out: per-particle loss
  int nslice, ngrid, nz, nphi, nmode;
  double rmax, ks, gammaz2, coef;  // coef = -2 Z0 k_s / (eev gamma_z^2)
};

__device__ __forceinline__ double block_sum_max(double v, double* sh, bool is_max) {
  // fixed order: warp xor tree, then one thread over the warp partials
  for (int o = 16; o > 0; o >>= 1) {
    const double t = __shfl_xor_sync(0xffffffffu, v, o);
    v = is_max ? fmax(v, t) : v + t;
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  double r = sh[0];
  for (int i = 1; i < (int)(blockDim.x >> 5); ++i) r = is_max ? fmax(r, sh[i]) : r + sh[i];
  return r;
}

// Cluster helpers: rank and size of the CTA's cluster, its hardware barrier,
// and loads of another CTA's shared memory.
__device__ __forceinline__ uint32_t cl_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cl_size() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cl_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}
__device__ __forceinline__ uint32_t cl_addr(const void* p, uint32_t rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(ptx::smem_u32(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ double cl_load(const double* p, uint32_t rank) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(cl_addr(p, rank)) : "memory");
  return v;
}
__device__ __forceinline__ double2 cl_load2(const double2* p, uint32_t rank) {
  double2 v;
  asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];"
               : "=d"(v.x), "=d"(v.y)
               : "r"(cl_addr(p, rank))
               : "memory");
  return v;
}
__device__ __forceinline__ longlong2 cl_load2(const longlong2* p, uint32_t rank) {
  longlong2 v;
  asm volatile("ld.shared::cluster.v2.s64 {%0, %1}, [%2];"
               : "=l"(v.x), "=l"(v.y)
               : "r"(cl_addr(p, rank))
               : "memory");
  return v;
}

// (c, s) = (c, s) times (a, b) as complex numbers
__device__ __forceinline__ void turn(double& c, double& s, double a, double b) {
  const double t = fma(c, a, -s * b);
  s = fma(s, a, c * b);
  c = t;
}

// A slice per cluster of C CTAs (C chosen so that the slices fill the GPU):
// each takes 1/C of the particles and of the modes.  Bound by the FP64 work per
// particle, done twice (radius and azimuth: a square root and two divisions; the
// phase: one sincos for all modes), and by the chain of the radial solves (one
// division per cell).  48 slices of 8192, nz = 2, |m| <= 1, 100 cells: 348 us
// with one CTA per slice, a sincos per harmonic, three divisions per cell and
// 64-bit shared atomics per particle; now 72 us, with the particles of a
// quiet-start beamlet adding theirs together (one slice 319 -> 63 us, 150 slices
// with one mode 160 -> 79, 250 slices with fifteen modes, one CTA each, 713 ->
// 267).
__global__ void __launch_bounds__(kScThreads) short_range_kernel(const ScArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double shd[kScThreads / 32];
  __shared__ double part[3];  // this CTA's sums of x and y, largest radius squared
  const int n = a.ngrid, nmode = a.nmode, nm = 2 * a.nphi + 1;
  longlong2* acc = reinterpret_cast<longlong2*>(smem);                    // [mode][cell]
  double2* u = reinterpret_cast<double2*>(acc + (size_t)nmode * n);       // [mode][cell]
  double* cp = reinterpret_cast<double*>(u + (size_t)nmode * n);          // Thomas c'
  const int tid = threadIdx.x, nt = blockDim.x, l = tid & 31;
  const int rank = (int)cl_rank(), C = (int)cl_size();
  for (int s = blockIdx.x / C; s < a.nslice; s += gridDim.x / C) {
    const int64_t q0 = a.off[s], np = a.off[s + 1] - q0;
    if (np <= 0) continue;  // uniform across the cluster
    // this CTA's particles, in whole groups of four
    const int64_t share = ((np + 3) / 4 + C - 1) / C * 4;
    const int64_t p0 = q0 + min(np, rank * share), p1 = q0 + min(np, (rank + 1) * share);
    const double eloss = a.eloss[s], cur = a.current[s];
    double sx = 0.0, sy = 0.0;
    for (int64_t p = p0 + tid; p < p1; p += nt) {
      sx += a.x[p];
      sy += a.y[p];
    }
    sx = block_sum_max(sx, shd, false);
    sy = block_sum_max(sy, shd, false);
    if (tid == 0) {
      part[0] = sx;
      part[1] = sy;
    }
    cl_sync();
    sx = sy = 0.0;
    for (int r = 0; r < C; ++r) {
      sx += cl_load(&part[0], r);
      sy += cl_load(&part[1], r);
    }
    const double xc = sx / (double)np, yc = sy / (double)np;
    double r2 = 0.0;
    for (int64_t p = p0 + tid; p < p1; p += nt) {
      const double dx = a.x[p] - xc, dy = a.y[p] - yc;
      r2 = fmax(r2, dx * dx + dy * dy);
    }
    r2 = block_sum_max(r2, shd, true);
    if (tid == 0) part[2] = r2;
    for (int i = tid; i < nmode * n; i += nt) acc[i] = make_longlong2(0, 0);
    cl_sync();
    for (int r = 0; r < C; ++r) r2 = fmax(r2, cl_load(&part[2], r));
    const double R = a.rmax * sqrt(r2);
    if (!(R > 0.0) || cur == 0.0) {
      for (int64_t p = p0 + tid; p < p1; p += nt) a.pez[p] = eloss;
      cl_sync();  // the next slice reuses the shared arrays
      continue;
    }
    const double dr = R / (double)n;
    // cell, e^{i phi} and e^{i theta} of a particle
    auto particle = [&](int64_t p, int& j, double& cph, double& sph, double& cth, double& sth) {
      const double dx = a.x[p] - xc, dy = a.y[p] - yc;
      const double r = sqrt(dx * dx + dy * dy);
      const double q = r / dr;  // NaN or beyond the wall: the last cell
      j = q >= 0.0 && q < (double)n ? (int)q : n - 1;
      const double ir = 1.0 / r;
      cph = r > 0.0 ? dx * ir : 1.0;
      sph = r > 0.0 ? dy * ir : 0.0;
      sincos(a.theta[p], &sth, &cth);
    };
    for (int64_t p = p0 + tid; p - l < p1; p += nt) {  // whole warps
      int j = -1;
      double cph = 0, sph = 0, cth = 0, sth = 0;
      if (p < p1) particle(p, j, cph, sph, cth, sth);
      // four consecutive particles of one cell add their sums together
      const int lead = __shfl_sync(0xffffffffu, j, l & ~3);
      const unsigned match = __ballot_sync(0xffffffffu, j >= 0 && j == lead);
      const bool same = ((match >> (l & ~3)) & 15u) == 15u;
      auto add = [&](longlong2* cell, double re, double im) {
        long long vr = __double2ll_rn(re * kScFix), vi = __double2ll_rn(im * kScFix);
        // lanes 0 and 1 of a group end with the sums of re and im
        const bool odd = (l & 1) != 0;
        long long v = (odd ? vi : vr) + __shfl_xor_sync(0xffffffffu, odd ? vr : vi, 1);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        unsigned long long* to = reinterpret_cast<unsigned long long*>(cell);
        if (same) {
          if ((l & 2) == 0) atomicAdd(to + (odd ? 1 : 0), (unsigned long long)v);
        } else if (j >= 0) {
          atomicAdd(to, (unsigned long long)vr);
          atomicAdd(to + 1, (unsigned long long)vi);
        }
      };
      double cl = cth, sl = sth;
      for (int h = 1; h <= a.nz; ++h) {
        longlong2* base = acc + ((size_t)(h - 1) * nm + a.nphi) * n + max(j, 0);
        add(base, cl, -sl);  // m = 0: e^{-i h theta}
        double pr = cl, pi = -sl, qr = cl, qi = -sl;
        for (int m = 1; m <= a.nphi; ++m) {
          // e^{-i(h theta + m phi)} and e^{-i(h theta - m phi)}
          turn(pr, pi, cph, -sph);
          turn(qr, qi, cph, sph);
          add(base + (size_t)m * n, pr, pi);
          add(base - (size_t)m * n, qr, qi);
        }
        turn(cl, sl, cth, sth);
      }
    }
    cl_sync();
    // this CTA's modes (t = rank, rank + C, ...): their sums over the cluster
    const int mine = (nmode - rank + C - 1) / C;
    const double rs = -kScUnfix / (6.283185307179586 * (double)np);
    for (int i = tid; i < mine * n; i += nt) {
      const int at = (rank + i / n * C) * n + i % n;
      long long re = 0, im = 0;
      for (int r = 0; r < C; ++r) {
        const longlong2 v = cl_load2(acc + at, r);
        re += v.x;
        im += v.y;
      }
      u[at] = make_double2(rs * (double)re, rs * (double)im);
    }
    __syncthreads();
    // one tridiagonal solve per mode (Thomas, FP64), in cell units of dr
    for (int k = tid; k < mine; k += nt) {
      const int t = rank + k * C, h = t / nm + 1, m = t % nm - a.nphi;
      const double kdr = (double)h * a.ks * dr;
      const double k2 = kdr * kdr / a.gammaz2;
      double2* ut = u + (size_t)t * n;
      double* ct = cp + (size_t)t * n;
      double prev_c = 0.0, prev_dr = 0.0, prev_di = 0.0;
      for (int j = 0; j < n; ++j) {
        const double rc = (double)j + 0.5;
        const double lo = (double)j, up = (double)(j + 1);
        const double diag = -lo - (j == n - 1 ? 2.0 * up : up) -
                            ((double)(m * m) / (rc * rc) + k2) * rc;
        const double2 b = ut[j];
        const double inv = 1.0 / (diag - lo * prev_c);
        prev_c = j < n - 1 ? up * inv : 0.0;
        prev_dr = (b.x - lo * prev_dr) * inv;
        prev_di = (b.y - lo * prev_di) * inv;
        ct[j] = prev_c;
        ut[j] = make_double2(prev_dr, prev_di);
      }
      for (int j = n - 2; j >= 0; --j) {
        const double2 nx = ut[j + 1];
        ut[j].x -= ct[j] * nx.x;
        ut[j].y -= ct[j] * nx.y;
      }
    }
    cl_sync();
    for (int i = tid; i < nmode * n; i += nt) {
      const int owner = i / n % C;
      if (owner != rank) u[i] = cl_load2(u + i, owner);
    }
    __syncthreads();
    const double scale = a.coef * cur;
    for (int64_t p = p0 + tid; p < p1; p += nt) {
      int j;
      double cph, sph, cth, sth;
      particle(p, j, cph, sph, cth, sth);
      double sum = 0.0, cl = cth, sl = sth;
      for (int h = 1; h <= a.nz; ++h) {
        const double2* base = u + ((size_t)(h - 1) * nm + a.nphi) * n + j;
        // Im[u_hm e^{i(h theta + m phi)}]
        double2 c = base[0];
        double im = c.x * sl + c.y * cl;
        double pr = cl, pi = sl, qr = cl, qi = sl;
        for (int m = 1; m <= a.nphi; ++m) {
          turn(pr, pi, cph, sph);
          turn(qr, qi, cph, -sph);
          c = base[(size_t)m * n];
          im += c.x * pi + c.y * pr;
          c = *(base - (size_t)m * n);
          im += c.x * qi + c.y * qr;
        }
        sum += (double)h * im;
        turn(cl, sl, cth, sth);
      }
      a.pez[p] = eloss + scale * sum;
    }
    cl_sync();  // the next slice reuses the shared arrays
  }
}

}  // namespace
}  // namespace g4b

using namespace g4b;

struct g4b_efield {
  g4b_ctx* ctx = nullptr;
  double rmax = 0, lambda = 0, ks = 0;
  int ngrid = 0, nz = 0, nphi = 0;
  size_t smem = 0;
  int resident[4] = {-1, -1, -1, -1};  // clusters of 1, 2, 4, 8 CTAs the GPU holds at once
};

namespace {
// Clusters the GPU holds at once: fewer than CTAs per SM times SMs over the size,
// for a cluster takes its SMs from one GPC.
int resident_clusters(g4b_efield* e) {
  for (int k = 0; k < 4 && e->resident[k] < 0; ++k) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1u << k);
    cfg.blockDim = dim3(kScThreads);
    cfg.dynamicSmemBytes = e->smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 1u << k;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    G4B_CUDA_TRY(cudaOccupancyMaxActiveClusters(&n, short_range_kernel, &cfg));
    e->resident[k] = std::max(1, n);
  }
  return G4B_OK;
}

int ensure_pez(g4b_beam* b) {
  if (b->d_pez) return G4B_OK;
  G4B_CUDA_TRY(dev_alloc(b->ctx, (void**)&b->d_pez,
                         (size_t)std::max<int64_t>(1, b->npart) * sizeof(double)));
  b->bytes += (uint64_t)std::max<int64_t>(1, b->npart) * sizeof(double);
  return G4B_OK;
}
}  // namespace

extern "C" {

int g4b_efield_create(g4b_ctx* c, double rmax, int ngrid, int nz, int nphi, double lambda,
                      g4b_efield** out) {
  if (!c || !out) return fail(G4B_ERR_ARG, "g4b_efield_create: null arg");
  if (ngrid < 0 || nz < 0 || nphi < 0 || !(lambda > 0.0) || !(rmax >= 0.0))
    return fail(G4B_ERR_ARG, "g4b_efield_create: bad parameters");
  const size_t nmode = (size_t)nz * (2 * nphi + 1);
  const size_t smem = nmode * (size_t)ngrid * (16 + 16 + 8);
  if (smem > 200u * 1024u)
    return fail(G4B_ERR_RANGE, "g4b_efield_create: nz*(2*nphi+1)*ngrid above 5120");
  g4b_efield* e = new (std::nothrow) g4b_efield();
  if (!e) return fail(G4B_ERR_NOMEM, "g4b_efield_create: host allocation");
  e->ctx = c;
  ctx_retain(c);
  e->rmax = rmax;
  e->ngrid = ngrid;
  e->nz = nz;
  e->nphi = nphi;
  e->lambda = lambda;
  e->ks = 4.0 * std::asin(1.0) / lambda;
  e->smem = smem;
  *out = e;
  return G4B_OK;
}

int g4b_efield_destroy(g4b_efield* e) {
  if (!e) return G4B_OK;
  ctx_release(e->ctx);
  delete e;
  return G4B_OK;
}

int g4b_efield_has_short_range(const g4b_efield* e) {
  return e && e->nz > 0 && e->ngrid > 0 && e->rmax > 0.0 ? 1 : 0;
}

int g4b_efield_short_range(g4b_efield* e, g4b_beam* b, double gammaz2) {
  if (!e || !b) return fail(G4B_ERR_ARG, "g4b_efield_short_range: null arg");
  if (b->precision != G4B_FP64)
    return fail(G4B_ERR_ARG, "g4b_efield_short_range: FP64 beam expected");
  if (b->ctx != e->ctx) return fail(G4B_ERR_ARG, "g4b_efield_short_range: contexts differ");
  if (!(gammaz2 > 0.0)) return fail(G4B_ERR_ARG, "g4b_efield_short_range: gammaz2 <= 0");
  if (!g4b_efield_has_short_range(e)) return G4B_OK;
  if (b->max_slice_np > kScMaxSliceNp)
    return fail(G4B_ERR_RANGE, "g4b_efield_short_range: more than 2^22 particles in a slice");
  g4b_ctx* c = b->ctx;
  G4B_CUDA_TRY(cudaSetDevice(c->device));
  if (int rc = ensure_pez(b)) return rc;
  b->use_pez = 1;
  if (b->npart == 0) return G4B_OK;
  ScArgs a{};
  a.x = b->x;
  a.y = b->y;
  a.theta = b->theta;
  a.off = b->d_off;
  a.current = b->d_current;
  a.eloss = b->d_eloss;
  a.pez = b->d_pez;
  a.nslice = b->nslice;
  a.ngrid = e->ngrid;
  a.nz = e->nz;
  a.nphi = e->nphi;
  a.nmode = e->nz * (2 * e->nphi + 1);
  a.rmax = e->rmax;
  a.ks = e->ks;
  a.gammaz2 = gammaz2;
  a.coef = -2.0 * kVacImp * e->ks / (kEev * gammaz2);
  G4B_CUDA_TRY(cudaFuncSetAttribute(short_range_kernel,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)e->smem));
  // the largest cluster of at least 512 particles per CTA with which the slices
  // still run at once (a slice more, and the last clusters run alone: 8192
  // particles with one mode, 55 slices in clusters of 8 / 4 82 / 52 us, 111 in 4 / 2
  // 99 / 71; one CTA per slice 139).  Where single CTAs take a second round, pairs
  // if that makes it shorter: large slices, the more of them the more CTAs share
  // an SM (200 slices of 8192 with 45 modes, one CTA per SM, 981 / 841 us; 600 of
  // 8192 with one mode, three, 266 / 246, but of 4096 137 / 153)
  if (int rc = resident_clusters(e)) return rc;
  const auto rounds = [&](int k) { return (b->nslice + e->resident[k] - 1) / e->resident[k]; };
  int C = 1;
  for (int k = 1; k < 4; ++k)
    if (rounds(k) == 1 && b->max_slice_np >= (512 << k)) C = 1 << k;
  if (rounds(0) == 2 && rounds(1) < 4 &&
      (int64_t)b->max_slice_np * c->sm_count >= (int64_t)2560 * e->resident[0])
    C = 2;
  const unsigned grid = (unsigned)(C * std::max(1, std::min(b->nslice, c->sm_count * 8)));
  {
    LaunchScope ls(c, "short_range");
    G4B_CUDA_TRY(launch_cluster(short_range_kernel, grid, kScThreads, (unsigned)C, e->smem,
                                c->stream, a));
  }
  return check_launch(c, "short_range_kernel");
}

int g4b_beam_set_particle_ez(g4b_beam* b, const double* ez) {
  if (!b) return fail(G4B_ERR_ARG, "g4b_beam_set_particle_ez: null beam");
  if (b->precision != G4B_FP64)
    return fail(G4B_ERR_ARG, "g4b_beam_set_particle_ez: FP64 beam expected");
  if (!ez) {
    b->use_pez = 0;
    return G4B_OK;
  }
  G4B_CUDA_TRY(cudaSetDevice(b->ctx->device));
  if (int rc = ensure_pez(b)) return rc;
  if (b->npart > 0) {
    G4B_CUDA_TRY(cudaMemcpyAsync(b->d_pez, ez, (size_t)b->npart * sizeof(double),
                                 cudaMemcpyHostToDevice, b->ctx->stream));
    G4B_CUDA_TRY(cudaStreamSynchronize(b->ctx->stream));
  }
  b->use_pez = 1;
  return G4B_OK;
}

int g4b_beam_get_particle_ez(g4b_beam* b, double* ez) {
  if (!b || !ez) return fail(G4B_ERR_ARG, "g4b_beam_get_particle_ez: null arg");
  if (!b->use_pez) return fail(G4B_ERR_STATE, "g4b_beam_get_particle_ez: no per-particle field");
  G4B_CUDA_TRY(cudaSetDevice(b->ctx->device));
  if (b->npart > 0) {
    G4B_CUDA_TRY(cudaMemcpyAsync(ez, b->d_pez, (size_t)b->npart * sizeof(double),
                                 cudaMemcpyDeviceToHost, b->ctx->stream));
  }
  G4B_CUDA_TRY(cudaStreamSynchronize(b->ctx->stream));
  return read_device_error(b->ctx, "g4b_beam_get_particle_ez");
}

}  // extern "C"
