// g4b_diag.cu -- per-slice beam and field diagnostics (DiagnosticCUDA) for sm_100a.
//
// A CTA reads its share of a slice's particles (or of the rows of its field
// plane) once and keeps every moment in registers; reductions run in a fixed
// order (warp xor tree, then warps in index order).  A slice is split over
// `parts` CTAs where there are fewer slices than the GPU holds CTAs; every CTA
// writes one record, and the host, which is what the results are for, adds the
// parts pairwise.  The entry points' records go straight to pinned host memory,
// a slice of one part in the caller's layout, so a call is one launch and one
// synchronisation.  A call, us, one CTA per slice with a device buffer and two or
// three copies to pageable memory -> now, beam / field: 1 slice of 8192 and 151^2
// 73 / 48 -> 32 / 25, 148 of 5000 and 129^2 65 / 47 -> 41 / 34, 1024 of 4096 and
// 101^2 126 / 102 -> 87 / 74, 4096 of 500 and 65^2 166 / 120 -> 123 / 109; 300 of
// 5000 with four harmonics 102 -> 75.  Bound by the latency of the loads and, with
// several harmonics, by the FP64 pipe.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <string>

#include "g4b_internal.cuh"

namespace g4b {

constexpr int kDiagThreads = 256;
constexpr int kDiagWarps = kDiagThreads / 32;
constexpr int kBeamDiagCtas = 2, kFieldDiagCtas = 8;  // per SM, before a slice is not split

enum class Red { Sum, Min, Max };

__device__ __forceinline__ double warp_red(double v, Red op) {
  for (int o = 16; o > 0; o >>= 1) {
    const double t = __shfl_xor_sync(0xffffffffu, v, o);
    v = op == Red::Sum ? v + t : (op == Red::Min ? fmin(v, t) : fmax(v, t));
  }
  return v;
}

struct BeamRecArgs {
  const int64_t* off;
  const double *x, *y, *px, *py, *gamma, *theta;
  // parts > 1: [nslice][parts][23 + 2 nharm]; else the caller's three arrays,
  // [nslice][23], then re and im [nslice][nharm] each
  double* rec;
  int nslice, nharm, need_aux, parts;
};

// g4_beam_slice_reduce_kernel (src/Core/DiagnosticCUDA.cpp:188-303); HP
// harmonics accumulated per pass over the particles, each by its own sincos
// corrected for the rounding of k theta.  Multiplying e^{i theta} up instead is
// a sincos for all, 300 slices of 5000 with four harmonics 36 us against 54, but
// its errors add up: at the eighth harmonic rms 1.3e-17 of the particles against
// 2.5e-18 (4.4e-18 without the correction, and 6e-16 at phases of 300).  More
// than four harmonics at once leave one CTA of registers per SM: 300 x 5000 with
// eight 126 us a call against 108.
template <int HP>
__global__ void __launch_bounds__(kDiagThreads, 2)
    beam_diag_kernel(const __grid_constant__ BeamRecArgs a) {
  constexpr int U = HP == 1 ? 4 : 2;  // particles in flight per thread
  __shared__ double part[kDiagWarps][23 + 2 * HP];
  ptx::pdl_wait();
  const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
  const int is = blockIdx.x / a.parts, ip = blockIdx.x % a.parts;
  const int64_t q0 = a.off[is], all = a.off[is + 1] - q0, per = (all + a.parts - 1) / a.parts;
  const int64_t p0 = q0 + min(all, ip * per), p1 = q0 + min(all, (ip + 1) * per);
  double v[23];
#pragma unroll
  for (int k = 0; k < 13; ++k) v[k] = 0.0;
  v[13] = 1.0e5; v[14] = -1.0e5;  // xmin xmax
  v[15] = 1.0e5; v[16] = -1.0e5;  // pxmin pxmax
  v[17] = 1.0e5; v[18] = -1.0e5;  // ymin ymax
  v[19] = 1.0e5; v[20] = -1.0e5;  // pymin pymax
  v[21] = 1.0e7; v[22] = 1.0;     // gmin gmax
  for (int hb = 0; hb < a.nharm; hb += HP) {
    const int hn = min(a.nharm - hb, HP);
    double br[HP], bi[HP];
#pragma unroll
    for (int h = 0; h < HP; ++h) br[h] = bi[h] = 0.0;
    for (int64_t pb = p0 + tid; pb < p1; pb += U * kDiagThreads) {
      double lx[U], ly[U], lpx[U], lpy[U], lg[U], lt[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t p = pb + u * kDiagThreads;
        if (p < p1) {
          lt[u] = a.theta[p];
          if (hb == 0) {
            lx[u] = a.x[p];
            ly[u] = a.y[p];
            lpx[u] = a.px[p];
            lpy[u] = a.py[p];
            lg[u] = a.gamma[p];
          }
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (pb + u * kDiagThreads >= p1) break;
        if (hb == 0) {
          const double xv = lx[u], yv = ly[u], pxv = lpx[u], pyv = lpy[u], gv = lg[u];
          v[0] += gv;
          v[1] += gv * gv;
          v[2] += xv;
          v[3] += xv * xv;
          v[4] += yv;
          v[5] += yv * yv;
          v[6] += pxv;
          v[7] += pxv * pxv;
          v[8] += pyv;
          v[9] += pyv * pyv;
          v[10] += xv * pxv;
          v[11] += yv * pyv;
          v[12] += 1.0;
          if (a.need_aux) {
            v[13] = fmin(v[13], xv); v[14] = fmax(v[14], xv);
            v[15] = fmin(v[15], pxv); v[16] = fmax(v[16], pxv);
            v[17] = fmin(v[17], yv); v[18] = fmax(v[18], yv);
            v[19] = fmin(v[19], pyv); v[20] = fmax(v[20], pyv);
            v[21] = fmin(v[21], gv); v[22] = fmax(v[22], gv);
          }
        }
#pragma unroll
        for (int h = 0; h < HP; ++h) {
          if (h >= hn) break;
          const double k = (double)(hb + h + 1), ph = k * lt[u];
          double err = fma(k, lt[u], -ph);  // of the product's rounding
          if (fabs(err) > 0x1p-27) err = 0.0;  // (phases above 2^26: as rounded)
          double sh, ch;
          sincos(ph, &sh, &ch);
          br[h] += fma(-err, sh, ch);
          bi[h] += fma(err, ch, sh);
        }
      }
    }
    if (hb == 0) {
#pragma unroll
      for (int k = 0; k < 23; ++k) {
        const Red op = k < 13 ? Red::Sum : ((k - 13) % 2 == 0 ? Red::Min : Red::Max);
        const double r = warp_red(v[k], op);
        if (l == 0) part[w][k] = r;
      }
    }
#pragma unroll
    for (int h = 0; h < HP; ++h) {
      if (h >= hn) break;
      const double rr = warp_red(br[h], Red::Sum), ri = warp_red(bi[h], Red::Sum);
      if (l == 0) {
        part[w][23 + 2 * h] = rr;
        part[w][24 + 2 * h] = ri;
      }
    }
    __syncthreads();
    if (tid < 23 + 2 * hn && (hb == 0 || tid >= 23)) {
      const int k = tid;
      const Red op = k < 13 || k >= 23 ? Red::Sum : ((k - 13) % 2 == 0 ? Red::Min : Red::Max);
      double r = part[0][k];
      for (int i = 1; i < kDiagWarps; ++i) {
        const double t = part[i][k];
        r = op == Red::Sum ? r + t : (op == Red::Min ? fmin(r, t) : fmax(r, t));
      }
      if (a.parts > 1) {
        a.rec[(size_t)blockIdx.x * (23 + 2 * a.nharm) + (k < 23 ? k : k + 2 * hb)] = r;
      } else if (k < 23) {
        a.rec[(size_t)is * 23 + k] = k >= 13 && !a.need_aux ? 0.0 : r;
      } else {
        double* b = a.rec + (size_t)a.nslice * (23 + (k % 2 ? 0 : a.nharm));
        b[(size_t)is * a.nharm + hb + (k - 23) / 2] = r;
      }
    }
    __syncthreads();
  }
}

// g4_field_slice_reduce_kernel (src/Core/DiagnosticCUDA.cpp:305-363): seven sums
// and the centre cell, [nslice][parts][7], then [nslice][2]; part ip takes the
// rows of its warps, parts * 8 rows apart.
template <typename C>
__global__ void __launch_bounds__(kDiagThreads)
    field_diag_kernel(int nslice, int n, int ld, int first, int parts, const C* cells,
                      double* rec) {
  __shared__ double part[kDiagWarps][7];
  ptx::pdl_wait();
  const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
  const int is0 = blockIdx.x / parts, ip = blockIdx.x % parts;
  const C* c = cells + (size_t)is0 * n * ld;
  const int is = (nslice + is0 - first) % nslice;
  const double shift = -0.5 * (double)(n - 1);
  double v[7] = {0, 0, 0, 0, 0, 0, 0};
  // a warp per row: coalesced row reads with no index division, the row's
  // sums first, then its y moments from the row's power
  for (int iy = ip * kDiagWarps + w; iy < n; iy += parts * kDiagWarps) {
    const C* row = c + (size_t)iy * ld;
    double p = 0, px = 0, pxx = 0, sre = 0, sim = 0;
#pragma unroll 4
    for (int ix = l; ix < n; ix += 32) {
      const C u = row[ix];
      const double re = u.x, im = u.y;
      const double wei = re * re + im * im;
      const double dx = (double)ix + shift;
      p += wei;
      px += dx * wei;
      pxx += dx * dx * wei;
      sre += re;
      sim += im;
    }
    const double dy = (double)iy + shift;
    v[0] += p;
    v[1] += px;
    v[2] += pxx;
    v[3] += dy * p;
    v[4] += dy * dy * p;
    v[5] += sre;
    v[6] += sim;
  }
#pragma unroll
  for (int k = 0; k < 7; ++k) {
    const double r = warp_red(v[k], Red::Sum);
    if (l == 0) part[w][k] = r;
  }
  __syncthreads();
  if (tid < 7) {
    double r = part[0][tid];
    for (int i = 1; i < kDiagWarps; ++i) r += part[i][tid];
    rec[((size_t)is * parts + ip) * 7 + tid] = r;
  } else if (tid == 32 && ip == 0) {
    const int ic = (n * n - 1) / 2;
    const C u = c[(size_t)(ic / n) * ld + (ic % n)];
    double* center = rec + (size_t)nslice * parts * 7 + 2 * (size_t)is;
    center[0] = u.x;
    center[1] = u.y;
  }
}

}  // namespace g4b

using namespace g4b;

namespace {
// Pinned host memory of the diagnostics entry points that kernels write to:
// one buffer per calling host thread (every call ends with a synchronisation,
// so it is free again for the thread's next one, on any device), as large as
// the thread's largest call, freed with the thread.
struct DiagHost {
  double* p = nullptr;
  size_t cap = 0;
  ~DiagHost() {
    if (p) cudaFreeHost(p);
  }
};
int diag_host(size_t n, double** out) {
  static thread_local DiagHost h;
  if (h.cap < n) {
    if (h.p) cudaFreeHost(h.p);
    h.p = nullptr;
    h.cap = 0;
    size_t cap = 8192;
    while (cap < n) cap *= 2;
    G4B_CUDA_TRY(cudaHostAlloc((void**)&h.p, cap * sizeof(double), cudaHostAllocPortable));
    h.cap = cap;
  }
  *out = h.p;
  return G4B_OK;
}

// CTAs per slice: `per_sm` CTAs on every SM, but no more than `most` (a share
// below which a CTA is not worth its launch).
int diag_parts(g4b_ctx* c, int nslice, int per_sm, int64_t most) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(most, per_sm * c->sm_count / nslice));
}
int field_parts(g4b_field* f) {
  return diag_parts(f->ctx, f->nslice, kFieldDiagCtas, (f->ngrid + 15) / 16);
}

int launch_field_diag(g4b_field* f, int parts, double* rec) {
  g4b_ctx* c = f->ctx;
  {
    LaunchScope ls(c, "diag_field");
    const unsigned grid = (unsigned)(f->nslice * parts);
    if (f->precision == G4B_FP64)
      G4B_CUDA_TRY(launch_pdl(field_diag_kernel<double2>, grid, kDiagThreads, 0, c->stream,
                              f->nslice, f->ngrid, f->ld, f->first, parts,
                              static_cast<const double2*>(f->a), rec));
    else
      G4B_CUDA_TRY(launch_pdl(field_diag_kernel<float2>, grid, kDiagThreads, 0, c->stream,
                              f->nslice, f->ngrid, f->ld, f->first, parts,
                              static_cast<const float2*>(f->a), rec));
  }
  return check_launch(c, "field_diag_kernel");
}

// Adds the first n values (N where it is known) of the parts' records of one
// slice into the first part's, pairwise: added one after another they would
// round as often as there are parts.
template <int N>
inline void add_parts(double* r, int parts, size_t stride, int n = N) {
  for (int d = 1; d < parts; d *= 2)
    for (int p = 0; p + d < parts; p += 2 * d) {
      double* __restrict__ a = r + p * stride;
      const double* __restrict__ b = a + d * stride;
      for (int k = 0; k < (N ? N : n); ++k) a[k] += b[k];
    }
}

size_t field_rec(int nslice, int parts) { return (size_t)nslice * (7 * parts + 2); }

// The field records into the caller's arrays; the parts' are overwritten.
void gather_field(double* rec, int nslice, int parts, double* stats, double* center) {
  if (parts == 1)
    std::memcpy(stats, rec, (size_t)nslice * 7 * sizeof(double));
  else
    for (int s = 0; s < nslice; ++s) {
      double* r = rec + (size_t)s * parts * 7;
      add_parts<7>(r, parts, 7);
      std::memcpy(stats + (size_t)s * 7, r, 7 * sizeof(double));
    }
  std::memcpy(center, rec + (size_t)nslice * parts * 7, (size_t)nslice * 2 * sizeof(double));
}
}  // namespace

namespace {

// ---- field diagnostics with fixed scratch ----------------------------------
// Some callers must not allocate device memory when they ask for the field
// statistics: a host that hands the device's memory to its own pool and
// forbids growth during a run, or a loop whose latency budget has no room for
// an allocation's implicit device-wide synchronisation.  For them the records of
// field_diag_kernel go to one fixed file-scope device array instead of the
// pinned buffer above, which grows with its thread's largest call.  Its size bounds the slices per call.
constexpr int kStaticDiagMaxSlices = 4096;               // 4096 x 9 doubles = 288 KiB
static __device__ __align__(256) double g_field_diag_scratch[kStaticDiagMaxSlices * 9];

constexpr int kStaticDiagMaxDevices = 64;
std::atomic<double*> g_field_diag_scratch_ptr[kStaticDiagMaxDevices];
std::mutex g_field_diag_scratch_mutex;

// Address of the array on `device` (which must be current).  The first call
// on a device asks the runtime for the symbol address (which may load the
// module); later calls read the cached pointer.
int static_diag_scratch(int device, double** out) {
  if (device < 0 || device >= kStaticDiagMaxDevices)
    return fail(G4B_ERR_RANGE, "g4b_diag_field_static: device index above 63");
  double* p = g_field_diag_scratch_ptr[device].load(std::memory_order_acquire);
  if (!p) {
    std::lock_guard<std::mutex> lock(g_field_diag_scratch_mutex);
    p = g_field_diag_scratch_ptr[device].load(std::memory_order_relaxed);
    if (!p) {
      const cudaError_t e = cudaGetSymbolAddress((void**)&p, g_field_diag_scratch);
      if (e != cudaSuccess) return cuda_fail(e, "g4b_diag_field_static: cudaGetSymbolAddress");
      g_field_diag_scratch_ptr[device].store(p, std::memory_order_release);
    }
  }
  *out = p;
  return G4B_OK;
}

}  // namespace

extern "C" {

int g4b_diag_beam(g4b_beam* b, int nharm, int need_aux, double* stats, double* bre,
                  double* bim) {
  if (!b || !stats || nharm < 1 || !bre || !bim)
    return fail(G4B_ERR_ARG, "g4b_diag_beam: bad argument");
  if (b->precision != G4B_FP64) return fail(G4B_ERR_ARG, "g4b_diag_beam: FP64 beam expected");
  g4b_ctx* c = b->ctx;
  G4B_CUDA_TRY(cudaSetDevice(c->device));
  const int ns = b->nslice, nrec = 23 + 2 * nharm;
  const int parts = diag_parts(c, ns, kBeamDiagCtas, (b->max_slice_np + 511) / 512);
  double* rec = nullptr;
  if (int rc = diag_host((size_t)ns * parts * nrec, &rec)) return rc;
  {
    LaunchScope ls(c, "diag_beam");
    const BeamRecArgs a{b->d_off, b->x, b->y,  b->px, b->py,    b->gamma,
                        b->theta, rec,  ns,    nharm, need_aux, parts};
    auto kern = nharm == 1 ? beam_diag_kernel<1> : beam_diag_kernel<4>;
    G4B_CUDA_TRY(launch_pdl(kern, (unsigned)(ns * parts), kDiagThreads, 0, c->stream, a));
  }
  if (int rc = check_launch(c, "beam_diag_kernel")) return rc;
  G4B_CUDA_TRY(cudaStreamSynchronize(c->stream));
  if (parts == 1) {
    const size_t nb = (size_t)ns * nharm;
    std::memcpy(stats, rec, (size_t)ns * 23 * sizeof(double));
    std::memcpy(bre, rec + (size_t)ns * 23, nb * sizeof(double));
    std::memcpy(bim, rec + (size_t)ns * 23 + nb, nb * sizeof(double));
    return G4B_OK;
  }
  for (int s = 0; s < ns; ++s) {
    double* r = rec + (size_t)s * parts * nrec;
    add_parts<13>(r, parts, nrec);
    add_parts<0>(r + 23, parts, nrec, 2 * nharm);
    for (int p = 1; p < parts; ++p) {
      const double* u = r + (size_t)p * nrec;
      for (int k = 13; k < 23; k += 2) {
        r[k] = std::fmin(r[k], u[k]);
        r[k + 1] = std::fmax(r[k + 1], u[k + 1]);
      }
    }
    std::memcpy(stats + (size_t)s * 23, r, 23 * sizeof(double));
    if (!need_aux) std::fill_n(stats + (size_t)s * 23 + 13, 10, 0.0);
    for (int h = 0; h < nharm; ++h) {
      bre[(size_t)s * nharm + h] = r[23 + 2 * h];
      bim[(size_t)s * nharm + h] = r[24 + 2 * h];
    }
  }
  return G4B_OK;
}

int g4b_diag_field(g4b_field* f, double* stats, double* center) {
  if (!f || !stats || !center) return fail(G4B_ERR_ARG, "g4b_diag_field: null arg");
  g4b_ctx* c = f->ctx;
  G4B_CUDA_TRY(cudaSetDevice(c->device));
  const int parts = field_parts(f);
  double* rec = nullptr;
  if (int rc = diag_host(field_rec(f->nslice, parts), &rec)) return rc;
  if (int rc = launch_field_diag(f, parts, rec)) return rc;
  G4B_CUDA_TRY(cudaStreamSynchronize(c->stream));
  gather_field(rec, f->nslice, parts, stats, center);
  return G4B_OK;
}

// Same statistics as g4b_diag_field, with the device scratch in a fixed
// file-scope array: nothing is allocated on the device or through the CUDA
// runtime's allocators.  Every scratch entry the call reads back is written
// by its own kernel first, so no part of the array has to start at zero.
int g4b_diag_field_static(g4b_field* f, double* stats, double* center) {
  if (!f || !stats || !center) return fail(G4B_ERR_ARG, "g4b_diag_field_static: null arg");
  if (f->nslice > kStaticDiagMaxSlices)
    return fail(G4B_ERR_RANGE, "g4b_diag_field_static: " + std::to_string(f->nslice) +
                                   " slices exceed the fixed scratch of " +
                                   std::to_string(kStaticDiagMaxSlices));
  g4b_ctx* c = f->ctx;
  G4B_CUDA_TRY(cudaSetDevice(c->device));
  double* rec = nullptr;
  if (int rc = static_diag_scratch(c->device, &rec)) return rc;
  // the records of every part fit: 7 nslice parts + 2 nslice <= 9 x 4096
  const int parts = std::min(field_parts(f), kStaticDiagMaxSlices / f->nslice);
  if (int rc = launch_field_diag(f, parts, rec)) return rc;
  const size_t n = field_rec(f->nslice, parts);
  const std::unique_ptr<double[]> host(new (std::nothrow) double[n]);
  if (!host) return fail(G4B_ERR_NOMEM, "g4b_diag_field_static: host allocation");
  G4B_CUDA_TRY(cudaMemcpyAsync(host.get(), rec, n * sizeof(double), cudaMemcpyDeviceToHost,
                               c->stream));
  G4B_CUDA_TRY(cudaStreamSynchronize(c->stream));
  gather_field(host.get(), f->nslice, parts, stats, center);
  return G4B_OK;
}

}  // extern "C"
