// g4b_adi.cu -- ADI field solver (FieldSolverADICUDA) for sm_100a.
//
// One field step = deposition + two fused half-step kernels:
//
//   pass X : for a band of W rows of one slice, 1-D bulk copies stage rows
//            r0-1 .. r0+W of the field and rows r0 .. r0+W-1 of the source in
//            shared memory; each warp forms R = u + i r d2y(u) + S for its row,
//            solves (1 - i r d2x) u' = R, and immediately forms the second
//            half-step's right-hand side R' = u' + i r d2x(u') + S (its
//            Laplacian runs along the row just solved).  R' is written
//            transposed ([slice][ix][iy]) through a TMA tensor store.
//   pass Y : each warp loads one contiguous row of R' (a column of the plane),
//            solves (1 - i r d2y) u'' = R' and writes u'' transposed back into
//            the natural layout.
//
// The tridiagonal system (1 - i r d2) u = R has constant coefficients, 1 + 2 i r
// on the diagonal and - i r beside it, and zero walls at k = -1 and k = n.
// With beta = (1 + 2 i r + sqrt(1 + 4 i r)) / 2 and q = i r / beta (|q| < 1) the
// matrix of the unbounded line factors into the two recurrences
//   y_k = (R_k + i r y_{k-1}) / beta,   u_k = y_k + q u_{k+1},
// the constant limit of the pivots of the reference's Thomas algorithm
// (src/Core/FieldSolverADICUDA.cpp:222-277).  Started with y_{-1} = 0 and
// u_n = 0 they satisfy every row but the wall at k = -1, which the homogeneous
// solution that vanishes at n mends:
//   u_k - u_0 (q^{k+2} - q^{2n+2-k}) / (1 - q^{2n+2}).
// A warp evaluates them: every lane runs the recurrences over its own M
// consecutive elements, the lane carries are combined by a Kogge-Stone scan of
// affine maps with multipliers q^(M 2^t) (only the steps whose multiplier is
// not zero at this precision: |q| is 0.02 at the configurations' r, so one step
// in place of four for FP32 rows of 201), and each lane adds its carry times a
// power of q.  All
// coefficients but the lanes' wall terms are the same in every lane: the
// single-run kernels read them from the constant bank.  With the Thomas pivots
// and the products of their factors in per-lane tables the passes spent as much
// of the load path on coefficients (four loads per element) as on the field:
// per pass X / Y of 1024 slices of 201^2 in FP32 152 / 136 -> 140 / 125 us (4.7
// and 5.3 TB/s of the field read and written), of 256 slices in FP64 96 / 83 ->
// 84 / 68 us, of 40 slices of 401^2 98 / 77 -> 90 / 70 us.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <limits>
#include <new>
#include <utility>
#include <vector>

#include <atomic>

#include "g4b_internal.cuh"

namespace g4b {

template <typename T> struct CT;
template <> struct CT<double> { using type = double2; };
template <> struct CT<float> { using type = float2; };

template <typename C>
__device__ __forceinline__ C cadd(C a, C b) { a.x += b.x; a.y += b.y; return a; }

// a + b*c
template <typename C>
__device__ __forceinline__ C cfma(C b, C c, C a) {
  C r;
  r.x = fma(b.x, c.x, fma(-b.y, c.y, a.x));
  r.y = fma(b.x, c.y, fma(b.y, c.x, a.y));
  return r;
}

// b*c with the fused roundings written out (the same bits in every kernel)
template <typename C>
__device__ __forceinline__ C cmul(C b, C c) {
  C r;
  r.x = fma(b.x, c.x, -(b.y * c.y));
  r.y = fma(b.x, c.y, b.y * c.x);
  return r;
}

// shuffles within groups of L lanes (L = 32: the warp; L = 16: its halves)
template <int L, typename C>
__device__ __forceinline__ C shfl_up_c(C v, int d) {
  v.x = __shfl_up_sync(0xffffffffu, v.x, d, L);
  v.y = __shfl_up_sync(0xffffffffu, v.y, d, L);
  return v;
}

template <int L, typename C>
__device__ __forceinline__ C shfl_down_c(C v, int d) {
  v.x = __shfl_down_sync(0xffffffffu, v.x, d, L);
  v.y = __shfl_down_sync(0xffffffffu, v.y, d, L);
  return v;
}


// ------------------------------------------------------ row arithmetic ---
// Forced inline into the single-run and the batched pass kernels: the same
// operations in the same order, hence the same bits, in every kernel.
// Pass X right-hand side of the band row at tile slot row + 1 (neighbours at
// slots row and row + 2): R = u + i r d2y(u) + S
// (src/Core/FieldSolverADICUDA.cpp:197-220); elements j >= jn are zero.
template <typename T, int M, typename C>
__device__ __forceinline__ void px_rhs(C (&v)[M], const C* tile, int ld, int row, int gl, int jn,
                                       T r, unsigned long long smask, const C* srow) {
#pragma unroll
  for (int j = 0; j < M; ++j) {
    const int k = gl * M + j;
    C R = C{0, 0};
    if (j < jn) {
      const C u = tile[(row + 1) * ld + k];
      const C up = tile[(row + 2) * ld + k];
      const C dn = tile[row * ld + k];
      const T lr = fma((T)-2, u.x, up.x + dn.x);
      const T li = fma((T)-2, u.y, up.y + dn.y);
      R.x = fma(-r, li, u.x);
      R.y = fma(r, lr, u.y);
      if ((smask >> j) & 1ull) R = cadd(R, srow[k]);
    }
    v[j] = R;
  }
}

// The row solve's coefficients: in the single-run kernels a parameter (operands
// from the constant bank), in the batched ones an image in global memory that
// differs from item to item.  There each is loaded where it is used (a
// broadcast from L1), volatile so that the compiler does not keep all M + 2
// powers in registers from their first use to their last: that spilled up to
// 1360 bytes per thread in pass Y.  Pass Y of 64 slices, us, plain loads -> now:
// 255^2 39 -> 25, 400^2 82 -> 60, 500^2 174 -> 90, 700^2 232 -> 145, 880^2 591 ->
// 314.
template <typename C>
struct RowParam {
  const RowConst<C>& k;
  __device__ __forceinline__ C P(int m) const { return k.P[m]; }
  __device__ __forceinline__ C A(int t) const { return k.A[t]; }
  __device__ __forceinline__ C cb() const { return k.cb; }
  __device__ __forceinline__ int nscan() const { return k.nscan; }
};
struct RowImage {
  const RowConst<float2>* k;
  static __device__ __forceinline__ float2 load(const float2* p) {
    float2 v;
    asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
  }
  __device__ __forceinline__ float2 P(int m) const { return load(&k->P[m]); }
  __device__ __forceinline__ float2 A(int t) const { return load(&k->A[t]); }
  __device__ __forceinline__ float2 cb() const { return load(&k->cb); }
  __device__ __forceinline__ int nscan() const { return __ldg(&k->nscan); }
};

// The tridiagonal solve (1 - i r d2) u = R of one row held by a group of L
// lanes, M consecutive elements each (lane gl: elements gl*M .. gl*M+M-1, of
// which the first jn lie in the row; R is zero in the others).  wall: the
// lanes' q^(gl M) / (1 - q^(2n+2)), then their q^(2n+2-(gl+1)M) / (1 - q^(2n+2)).
template <typename T, int M, int L, typename C, typename KC>
__device__ __forceinline__ void row_solve(C (&v)[M], const KC K, const C* wall, int gl, int jn,
                                          T r) {
  constexpr int kScan = L == 32 ? 5 : 4;  // log2 L
  const C we = wall[gl], wd = wall[L + gl];
  const C cb = K.cb();
  v[0] = cmul(cb, v[0]);
#pragma unroll
  for (int j = 1; j < M; ++j) {
    C t;
    t.x = fma(-r, v[j - 1].y, v[j].x);
    t.y = fma(r, v[j - 1].x, v[j].y);
    v[j] = cmul(cb, t);
  }
  C b = v[M - 1];
#pragma unroll
  for (int t = 0; t < kScan; ++t) {
    if (t >= K.nscan()) break;
    const C o = shfl_up_c<L>(b, 1 << t);
    if (gl >= 1 << t) b = cfma(K.A(t), o, b);
  }
  C yin = shfl_up_c<L>(b, 1);
  if (gl == 0) yin = C{0, 0};
#pragma unroll
  for (int j = 0; j < M; ++j) v[j] = cfma(K.P(j + 1), yin, v[j]);
  if (jn < M) {  // u is zero from n on
#pragma unroll
    for (int j = 0; j < M; ++j)
      if (j >= jn) v[j] = C{0, 0};
  }
  const C q = K.P(1);
#pragma unroll
  for (int j = M - 2; j >= 0; --j) v[j] = cfma(q, v[j + 1], v[j]);
  b = v[0];
#pragma unroll
  for (int t = 0; t < kScan; ++t) {
    if (t >= K.nscan()) break;
    const C o = shfl_down_c<L>(b, 1 << t);
    if (gl + (1 << t) < L) b = cfma(K.A(t), o, b);
  }
  C uin = shfl_down_c<L>(b, 1);
  if (gl == L - 1) uin = C{0, 0};
  // the wall at k = -1, from lane 0's first element
  C u0 = cfma(K.P(M), uin, v[0]);
  u0.x = -__shfl_sync(0xffffffffu, u0.x, 0, L);
  u0.y = -__shfl_sync(0xffffffffu, u0.y, 0, L);
  const C c = cmul(we, u0);
  uin.x -= fma(wd.x, u0.x, -(wd.y * u0.y));
  uin.y -= fma(wd.x, u0.y, wd.y * u0.x);
#pragma unroll
  for (int j = 0; j < M; ++j) v[j] = cfma(K.P(j + 2), c, cfma(K.P(M - j), uin, v[j]));
}

// R' = u' + i r d2x(u') + S (src/Core/FieldSolverADICUDA.cpp:279-323) of a
// solved row, in place with the original left neighbour carried along.
template <typename T, int M, int L, typename C>
__device__ __forceinline__ void px_rprime(C (&v)[M], int gl, T r, unsigned long long smask,
                                          const C* srow) {
  C prev = shfl_up_c<L>(v[M - 1], 1);
  if (gl == 0) prev = C{0, 0};
  C right = shfl_down_c<L>(v[0], 1);
  if (gl == L - 1) right = C{0, 0};
#pragma unroll
  for (int j = 0; j < M; ++j) {
    const int k = gl * M + j;
    const C cur = v[j];
    const C upp = j < M - 1 ? v[j + 1] : right;
    const T lr = fma((T)-2, cur.x, upp.x + prev.x);
    const T li = fma((T)-2, cur.y, upp.y + prev.y);
    C R;
    R.x = fma(-r, li, cur.x);
    R.y = fma(r, lr, cur.y);
    if ((smask >> j) & 1ull) R = cadd(R, srow[k]);
    v[j] = R;
    prev = cur;
  }
}

// Warps per CTA and CTAs per SM (launch bounds) of the ADI kernels: FP64 9
// warps of 32-lane rows, three CTAs per SM up to M = 7 (ngrid 224: pass X's
// three tiles still fit the SM's shared memory); FP32 10 warps of 32-lane rows or 5 warps of two
// 16-lane rows each (10 rows per band either way; smaller CTAs of 16-lane
// rows keep six on an SM so that one CTA's loads and stores overlap the
// others' solves).  FP32 rows of 32 x 33 get the registers of one CTA per SM:
// at 96 the batched form spills (64 slices of 880^2, X / Y: 387 / 326 -> 373 /
// 314 us).
template <typename T, int L> struct BandW {
  static constexpr int value = sizeof(T) == 8 ? 9 : (L == 16 ? 5 : 10);
};
template <typename T, int M, int L> struct AdiBlocks {
  static constexpr int value =
      sizeof(T) == 8 ? (M <= 7 ? 3 : 2)
                     : (L == 16 ? (M <= 9 ? 8 : (M <= 17 ? 6 : 4))
                                : (M <= 9 ? 4 : (M <= 25 ? 2 : 1)));
};

// One band of W rows (pass X) or W transposed columns (pass Y) of slice s.
// A row is solved by L lanes holding M elements each: L = 32, one row per
// warp; L = 16, two rows per warp (one per half), for rows that fit 16 M
// slots more closely than 32 M.  bar is an initialised mbarrier; parity the
// phase this band waits on.  Returns false, with nothing solved or stored, if
// the band's rows did not arrive within the bounded wait (the device error
// flag then says so); the result is the same in every thread of the CTA.
template <typename T, int M, bool PX, int L, typename KC>
__device__ __forceinline__ bool adi_band(const AdiPassArgs& a, const KC K,
                                         const CUtensorMap* tm_out, int s, int band,
                                         unsigned char* smem, uint64_t* bar, uint32_t parity) {
  using C = typename CT<T>::type;
  constexpr int R = 32 / L;                     // rows per warp
  constexpr int W = BandW<T, L>::value * R;     // rows per band
  const int n = a.n, ld = a.ld;
  const int r0 = band * W;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int gl = lane & (L - 1);                // lane within the row's group
  const int row = warp * R + (lane >> 4) * (R - 1);  // row within the band
  constexpr int kTileRows = PX ? W + 2 : W;
  const bool has_src = PX && a.src != nullptr;

  C* tile = reinterpret_cast<C*>(smem);
  C* stile = tile + kTileRows * ld;
  C* out = reinterpret_cast<C*>(smem + a.out_off);
  __shared__ double dpart[PX ? 1 : W][9];  // pass Y: per-row diagnostic partials

  const size_t plane = (size_t)n * ld;
  const int lo = PX ? max(r0 - 1, 0) : r0;
  const int hi = PX ? min(r0 + W, n - 1) : min(r0 + W - 1, n - 1);
  const int slot0 = PX ? lo - (r0 - 1) : 0;
  // the source is non-zero only on the slice's tile: rows [sy0, sy0+sbh),
  // columns [sx0, sx0+sbw); stile holds the tile rows of this band.  The
  // descriptor is written by the deposition, which may still be draining
  // when this kernel starts (launch_pdl): a plain load, which stays after
  // ptx::pdl_wait, not a read-only-path load the compiler may issue earlier
  const int4 sd = has_src ? a.desc[s] : make_int4(0, 0, 0, 0);
  const int sx0 = sd.x, sbw = sd.z;
  const int srow_lo = max(r0, sd.y);
  const int srow_hi = min(min(r0 + W, n), sd.y + sd.w);
  const bool band_src = has_src && sbw > 0 && srow_lo < srow_hi;
  if (tid == 0) {
    const C* in = reinterpret_cast<const C*>(a.in) + (size_t)s * plane;
    const uint32_t bytes_in = (uint32_t)((hi - lo + 1) * ld * sizeof(C));
    const uint32_t bytes_s =
        band_src ? (uint32_t)((srow_hi - srow_lo) * sbw * sizeof(C)) : 0u;
    ptx::mbar_expect_tx(bar, bytes_in + bytes_s);
    ptx::bulk_g2s(tile + slot0 * ld, in + (size_t)lo * ld, bytes_in, bar);
    if (band_src) {
      const C* sp = reinterpret_cast<const C*>(a.src) + (size_t)s * a.src_cap +
                    (size_t)(srow_lo - sd.y) * sbw;
      ptx::bulk_g2s(stile + (srow_lo - r0) * sbw, sp, bytes_s, bar);
    }
  }
  if (PX) {
    // rows outside the plane are the zero Dirichlet halo (missing neighbour
    // is zero, src/Core/FieldSolverADICUDA.cpp:197-207)
    for (int t = 0; t < kTileRows; ++t) {
      const int g = r0 - 1 + t;
      if (g < 0 || g > n - 1)
        for (int k = tid; k < ld; k += blockDim.x) tile[t * ld + k] = C{0, 0};
    }
  }
  const bool arrived = ptx::mbar_wait_bounded(bar, parity, a.err);
  if (!__syncthreads_and(arrived)) return false;
  const T r = (T)a.r;
  const int iy = r0 + row;
  const bool active = iy < n;
  const bool row_src = band_src && iy >= srow_lo && iy < srow_hi;
  const C* srow = stile + row * sbw - sx0;  // srow[k] for k in [sx0, sx0+sbw)
  // bit j set: this lane's element j lies in the source tile's columns
  unsigned long long smask = 0ull;
  if (row_src) {
    const int jlo = min(max(sx0 - gl * M, 0), M), jhi = min(max(sx0 + sbw - gl * M, 0), M);
    smask = ((1ull << jhi) - 1ull) & ~((1ull << jlo) - 1ull);
  }
  // elements j < jn lie in the row (none for a row past the plane)
  const int jn = active ? min(max(n - gl * M, 0), M) : 0;
  C v[M];

  // a warp with any row in the plane solves both (a row past the plane is
  // all zeros), so that every lane takes part in the group shuffles
  if (__any_sync(0xffffffffu, active)) {
    if (PX) {
      px_rhs<T, M>(v, tile, ld, row, gl, jn, r, smask, srow);
    } else {
#pragma unroll
      for (int j = 0; j < M; ++j) v[j] = j < jn ? tile[row * ld + gl * M + j] : C{0, 0};
    }
    row_solve<T, M, L>(v, K, reinterpret_cast<const C*>(static_cast<const RowConst<C>*>(a.tab) + 1),
                       gl, jn, r);
    if (PX) px_rprime<T, M, L>(v, gl, r, smask, srow);
  } else {
#pragma unroll
    for (int j = 0; j < M; ++j) v[j] = C{0, 0};
  }

  if (!PX && a.zero_count > 0) {
    const int zs = (s - a.zero_start + a.nslice) % a.nslice;
    if (zs < a.zero_count) {
#pragma unroll
      for (int j = 0; j < M; ++j) v[j] = C{0, 0};
    }
  }
  if (!PX && a.diag != nullptr) {
    // field diagnostics of this band (g4_field_slice_reduce_kernel,
    // src/Core/DiagnosticCUDA.cpp:305-363): this lane group holds column
    // ix = r0 + row, rows iy = gl*M + j of the solved plane
    // each lane sums its M cells in the state precision T (exact cell
    // offsets; partials of <= 33 terms, rounding at the level of the state's
    // own); the lanes of a column add in FP64 (<= 32 terms); the power and
    // the other sums of the band's warps and (in the finalize) of the bands
    // are added with compensation (csum_*), as are the slices on the host
    const T shift = (T)(-0.5 * (double)(n - 1));
    const double dx = (double)iy + (double)shift;  // iy is the column index in pass Y
    T tp = 0, ty1 = 0, ty2 = 0, tre = 0, tim = 0;
    double cre = 0, cim = 0;
    const int ic = (n * n - 1) / 2;
    const int icy = ic / n, icx = ic - icy * n;
    if (active) {
      if (jn < M) {  // cells past the row end
#pragma unroll
        for (int j = 0; j < M; ++j)
          if (j >= jn) v[j] = C{0, 0};
      }
      const T dy0 = (T)(gl * M) + shift;  // exact: small integers and halves
#pragma unroll
      for (int j = 0; j < M; ++j) {
        const T re = v[j].x, im = v[j].y;
        const T wei = fma(re, re, im * im);
        const T dy = dy0 + (T)j;
        tp += wei;
        ty1 = fma(dy, wei, ty1);
        ty2 = fma(dy * dy, wei, ty2);
        tre += re;
        tim += im;
      }
      const int jc = iy == icx ? icy - gl * M : -1;
      if (jc >= 0 && jc < M) {
#pragma unroll
        for (int j = 0; j < M; ++j)
          if (j == jc) {
            cre = (double)v[j].x;
            cim = (double)v[j].y;
          }
      }
    }
    // power over the column in FP64; the moments and sums over the column's
    // lanes in the state precision; the x moments follow from the column's
    // power (x is the column); the centre cell comes from the one lane that
    // holds it
    double sp = (double)tp;
    for (int o = L / 2; o > 0; o >>= 1) sp += __shfl_xor_sync(0xffffffffu, sp, o);
    T vals[4] = {ty1, ty2, tre, tim};
#pragma unroll
    for (int q = 0; q < 4; ++q)
      for (int o = L / 2; o > 0; o >>= 1) vals[q] += __shfl_xor_sync(0xffffffffu, vals[q], o);
    if (gl == 0) {
      dpart[row][0] = sp;
      dpart[row][1] = dx * sp;
      dpart[row][2] = dx * dx * sp;
      dpart[row][3] = (double)vals[0];
      dpart[row][4] = (double)vals[1];
      dpart[row][5] = (double)vals[2];
      dpart[row][6] = (double)vals[3];
      dpart[row][7] = 0.0;
      dpart[row][8] = 0.0;
    }
    __syncwarp();
    if (cre != 0.0 || cim != 0.0) {  // the lane holding the centre cell
      dpart[row][7] = cre;
      dpart[row][8] = cim;
    }
  }
  if (PX) __syncthreads();  // out overlays the input tile
#pragma unroll
  for (int j = 0; j < M; ++j) {
    const int k = gl * M + j;
    if (j < jn) out[k * W + row] = v[j];
  }
  ptx::fence_proxy_async();
  __syncthreads();  // the staged rows and the diagnostic partials are complete
  if (tid == 0) {
    for (int i = 0; i < a.nbox; ++i)
      ptx::tma_store_3d(tm_out, out + (size_t)i * a.box_rows * W, 2 * r0,
                        i * a.box_rows, s);
    ptx::bulk_commit();
  }
  // the band's diagnostic sums, over its rows in order, while the stores run
  if (!PX && a.diag != nullptr && tid >= 32 && tid < 32 + 9) {
    const int q = tid - 32;
    double t = dpart[0][q], tc = 0.0;
    for (int w = 1; w < W; ++w) ptx::csum_add(t, tc, dpart[w][q]);
    a.diag[((size_t)s * a.nband + band) * 9 + q] = t + tc;
  }
  if (tid == 0) ptx::bulk_wait_read0();
  return true;
}

template <typename T, int M, bool PX, int L>
__global__ void __launch_bounds__(BandW<T, L>::value * 32, AdiBlocks<T, M, L>::value)
    adi_pass_kernel(const __grid_constant__ AdiPassArgs a,
                    const __grid_constant__ RowConst<typename CT<T>::type> K,
                    const __grid_constant__ CUtensorMap tm_out) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    ptx::mbar_init(&bar, 1);
    ptx::fence_mbar_init();
  }
  __syncthreads();
  ptx::pdl_wait();
  adi_band<T, M, PX, L>(a, RowParam<typename CT<T>::type>{K}, &tm_out, blockIdx.x / a.nband,
                        blockIdx.x % a.nband, smem, &bar, 0u);
}

// Persistent form over a work list of (run, slice, band) items of many runs
// (one mbarrier, one phase per item; tensor maps read from global memory).
template <typename T, int M, bool PX, int L>
__global__ void __launch_bounds__(BandW<T, L>::value * 32, AdiBlocks<T, M, L>::value)
    adi_batch_kernel(const __grid_constant__ AdiBatchArgs b) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    ptx::mbar_init(&bar, 1);
    ptx::fence_mbar_init();
  }
  __syncthreads();
  const int nitems = *b.nitems;
  uint32_t parity = 0;
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const int4 w = b.items[it];
    const CUtensorMap* tm = b.maps + w.x;
    if (threadIdx.x == 0) ptx::fence_tensormap_acquire(tm);
    // a band whose rows never arrived leaves the barrier's phase open: stop
    // (the error flag reports it) rather than wait on it again
    const AdiPassArgs& a = b.args[w.x];
    const RowImage K{static_cast<const RowConst<float2>*>(a.tab)};
    if (!adi_band<T, M, PX, L>(a, K, tm, w.y, w.z, smem, &bar, parity)) return;
    parity ^= 1u;
    __syncthreads();
  }
}

// ------------------------------------------------------------ deposition ---
// Deterministic replacement of adi_zero_source_grid + adi_deposit_source_atomic
// (src/Core/FieldSolverADICUDA.cpp:98-174).  One CTA per beam slice:
//  1. a pass over the slice's particles finds a bound q of the per-particle
//     weights sqrt(faw2)/gamma and the bounding box of the touched cells;
//  2. the box is accumulated in shared memory as int64 fixed point with the
//     exponent 2^E chosen so that count * q * 2^E < 2^62 (integer adds are
//     associative, so the result does not depend on the order of the atomics);
//  3. the CTA writes only the box, scl * sum * 2^-E, as a compact tile of the
//     target slice, and the tile's (x0, y0, width, height) descriptor; the
//     source is zero outside the box.  Boxes larger than the shared-memory
//     accumulator are done in row bands.
struct DepositArgs {
  const double *x, *y, *gamma, *theta;
  const int64_t* off;
  const double* current;
  double fc, xks, delz, vacimp, eev;
  double2* src;        // compact tiles, src_cap cells per slice
  int4* desc;          // per target slice
  size_t src_cap;
  int nslice, n, ld, first, harm, acc_cells;
  double gridmax, dgrid, inv_dgrid, ax, ay, kx, ky, gradx, grady;
  int* err;
};

// x / dgrid by the reciprocal and one Newton correction of the quotient.
__device__ __forceinline__ double dep_over_dgrid(const DepositArgs& a, double x) {
  const double t = x * a.inv_dgrid;
  return fma(fma(-t, a.dgrid, x), a.inv_dgrid, t);
}

__device__ __forceinline__ bool dep_cell(const DepositArgs& a, double xp, double yp,
                                         int& ix, int& iy, double& wx, double& wy) {
  if (!(xp > -a.gridmax && xp < a.gridmax && yp > -a.gridmax && yp < a.gridmax))
    return false;
  const double wx_raw = dep_over_dgrid(a, xp + a.gridmax);
  const double wy_raw = dep_over_dgrid(a, yp + a.gridmax);
  ix = (int)floor(wx_raw);
  iy = (int)floor(wy_raw);
  if (ix < 0 || ix >= a.n - 1 || iy < 0 || iy >= a.n - 1) return false;
  wx = 1.0 + (double)ix - wx_raw;
  wy = 1.0 + (double)iy - wy_raw;
  return true;
}

// The particle's charge weight is sqrt(faw2) / gamma.
__device__ __forceinline__ double dep_faw2(const DepositArgs& a, double xp, double yp) {
  const double dx = xp - a.ax, dy = yp - a.ay;
  return 1.0 + a.kx * dx * dx + a.ky * dy * dy + 2.0 * (a.gradx * dx + a.grady * dy);
}

// What the first pass keeps of the particles in the grid: the largest faw2, the
// smallest |gamma|, the box of their base cells and their number.
struct DepBox {
  double fmx = 0.0, gmn = INFINITY;
  int ixmin = 1 << 30, iymin = 1 << 30, ixmax = -1, iymax = -1, cnt = 0;
  __device__ __forceinline__ void warp_reduce() {
    for (int o = 16; o > 0; o >>= 1) {
      const double f = __shfl_xor_sync(0xffffffffu, fmx, o), g = __shfl_xor_sync(0xffffffffu, gmn, o);
      fmx = f > fmx ? f : fmx;
      gmn = g < gmn ? g : gmn;
    }
    ixmin = __reduce_min_sync(0xffffffffu, ixmin);
    iymin = __reduce_min_sync(0xffffffffu, iymin);
    ixmax = __reduce_max_sync(0xffffffffu, ixmax);
    iymax = __reduce_max_sync(0xffffffffu, iymax);
    cnt = __reduce_add_sync(0xffffffffu, cnt);
  }
};

constexpr int kDepFp64U = 2;  // particles in flight per thread (the first pass)
// One CTA of 1024 threads per SM with a band of 12800 cells: tiles of 80-110
// cells a side are one band, so a particle's cell, weight and phase are worked
// out once (two 512-thread CTAs with bands of 6144 cells: twice the cells and
// the first pass's divisions; us per launch with 256 slices of 8192 at 201^2:
// 94 -> 66, 64 slices of 4096 at 255^2 48 -> 30, 40 slices of 4096 at 401^2 80 ->
// 48, 1 slice of 8192 at 151^2 37 -> 29, 8 of 2048 at 101^2 17 -> 15).  Bound by
// the FP64 chain of a particle: sincos, square root, division.  A few slices as
// clusters of CTAs, their tiles added through distributed shared memory, gain a
// tenth at 4 slices and lose as much at 16 and with small slices.
constexpr int kDepFp64Threads = 1024;
constexpr size_t kDepFp64Acc = 200 * 1024;  // accumulators: 12800 cells, one band in most runs

__global__ void __launch_bounds__(kDepFp64Threads, 1) deposit_slice_kernel(const DepositArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ double shd[2][32];
  __shared__ int shi[5][32];
  ptx::pdl_wait();
  unsigned long long* acc = reinterpret_cast<unsigned long long*>(smem);
  const int bs = blockIdx.x;
  const int tid = threadIdx.x;
  const int target = (bs + a.first) % a.nslice;
  double2* S = a.src + (size_t)target * a.src_cap;
  const int64_t p0 = a.off[bs], p1 = a.off[bs + 1];
  // adi_compute_slice_scl (src/Core/FieldSolverADICUDA.cpp:75-96); a kernel of
  // its own was 2 us of a step's launches
  double scl = 0.0;
  if (p1 > p0) {
    scl = a.fc * a.vacimp * a.current[bs] * a.xks * a.delz;
    scl /= 4.0 * a.eev * (double)(p1 - p0) * a.dgrid * a.dgrid;
  }

  // largest faw2 and smallest |gamma|: the weights are at most sqrt(fmx) / gmn
  DepBox m;
  const int nt = blockDim.x;
  if (scl != 0.0) {
    // kDepFp64U particles in flight per thread: their loads are issued
    // before any of them is processed
    for (int64_t pb = p0 + tid; pb < p1; pb += (int64_t)kDepFp64U * nt) {
      double lx[kDepFp64U], ly[kDepFp64U], lg[kDepFp64U];
#pragma unroll
      for (int u = 0; u < kDepFp64U; ++u) {
        const int64_t p = pb + (int64_t)u * nt;
        if (p < p1) {
          lx[u] = a.x[p];
          ly[u] = a.y[p];
          lg[u] = a.gamma[p];
        }
      }
#pragma unroll
      for (int u = 0; u < kDepFp64U; ++u) {
        if (pb + (int64_t)u * nt >= p1) break;
        int ix, iy;
        double wx, wy;
        if (!dep_cell(a, lx[u], ly[u], ix, iy, wx, wy)) continue;
        const double f = dep_faw2(a, lx[u], ly[u]), g = fabs(lg[u]);
        m.fmx = f > m.fmx ? f : m.fmx;
        m.gmn = g < m.gmn ? g : m.gmn;
        if (!(f >= 0.0 && g > 0.0)) m.fmx = INFINITY;  // no finite weight
        m.ixmin = min(m.ixmin, ix);
        m.ixmax = max(m.ixmax, ix);
        m.iymin = min(m.iymin, iy);
        m.iymax = max(m.iymax, iy);
        ++m.cnt;
      }
    }
  }
  // one exchange through shared memory, then the same tree in every warp (seven
  // block reductions, each a serial loop over 32 warps: 6 us more of a launch)
  const int w = tid >> 5, l = tid & 31;
  m.warp_reduce();
  if (l == 0) {
    shd[0][w] = m.fmx;
    shd[1][w] = m.gmn;
    shi[0][w] = m.ixmin;
    shi[1][w] = m.iymin;
    shi[2][w] = m.ixmax;
    shi[3][w] = m.iymax;
    shi[4][w] = m.cnt;
  }
  __syncthreads();
  if (l < (nt >> 5)) {
    m.fmx = shd[0][l];
    m.gmn = shd[1][l];
    m.ixmin = shi[0][l];
    m.iymin = shi[1][l];
    m.ixmax = shi[2][l];
    m.iymax = shi[3][l];
    m.cnt = shi[4][l];
  } else {
    m.cnt = 0;  // lane 0's values are copies of this warp's: they add no extreme
  }
  m.warp_reduce();
  double qmax = sqrt(m.fmx) / m.gmn;
  if (!(qmax <= 1e300)) qmax = INFINITY;  // taken up to there (m.gmn infinite: no charge)

  const bool any = m.cnt > 0 && qmax > 0.0;
  if (any && !(qmax < INFINITY) && tid == 0) atomicOr(a.err, kErrFixedRange);
  const bool ok = any && qmax < INFINITY;
  int bx0 = 0, by0 = 0, bw = 0, bh = 0;
  double scale = 0.0, unscale = 0.0;
  if (ok) {
    bx0 = m.ixmin;
    by0 = m.iymin;
    bw = m.ixmax - m.ixmin + 2;  // corners ix..ix+1
    bh = m.iymax - m.iymin + 2;
    int e;
    frexp(qmax * (double)m.cnt, &e);  // qmax*m.cnt < 2^e
    scale = ldexp(1.0, 62 - e);
    unscale = scl * ldexp(1.0, e - 62);
  }
  if (tid == 0) a.desc[target] = make_int4(bx0, by0, ok ? bw : 0, bh);
  if (!ok) return;
  const int band_h = max(1, min(bh, a.acc_cells / bw));
  const double hphase = (double)a.harm;

  for (int yb = by0; yb < by0 + bh; yb += band_h) {
    const int hb = min(band_h, by0 + bh - yb);
    // four 32-bit planes per band: low and high words of the real and the
    // imaginary 64-bit sums (a 64-bit shared atomic costs about four 32-bit
    // ones; the low word's carry goes to the high word, so every sum is the
    // exact 64-bit integer whatever the order of the adds)
    const int ncell = hb * bw;
    unsigned int* lre = reinterpret_cast<unsigned int*>(acc);
    unsigned int* lim = lre + ncell;
    int* hre = reinterpret_cast<int*>(lim + ncell);
    int* him = hre + ncell;
    for (int i = tid; i < 2 * ncell; i += blockDim.x) acc[i] = 0ull;
    __syncthreads();
    auto add = [&](int cell, long long cr, long long ci) {
      const unsigned int rlo = (unsigned int)cr, ilo = (unsigned int)ci;
      const unsigned int rold = atomicAdd(&lre[cell], rlo);
      const unsigned int iold = atomicAdd(&lim[cell], ilo);
      atomicAdd(&hre[cell], (int)(cr >> 32) + (rold + rlo < rold ? 1 : 0));
      atomicAdd(&him[cell], (int)(ci >> 32) + (iold + ilo < iold ? 1 : 0));
    };
    // One particle per lane, the next one's loads in flight.  Four consecutive
    // particles of one base cell (a quiet-start beamlet: nbins = 4 particles at
    // one transverse position) are summed over their lanes, each of which adds
    // one corner (the same integer sums by a quarter of the atomics).
    const int64_t np = p1 - p0;
    double nx = 0, ny = 0, ng = 1, nt_ = 0;
    auto load = [&](int64_t p) {
      if (p < np) {
        nx = a.x[p0 + p];
        ny = a.y[p0 + p];
        ng = a.gamma[p0 + p];
        nt_ = a.theta[p0 + p];
      }
    };
    load(tid);
    for (int64_t p = tid; p - l < np; p += nt) {  // whole warps
      const double xp = nx, yp = ny, gp = ng, tp = nt_;
      load(p + nt);
      int cid = -1, ix, iy;  // (ext row iy - yb + 1, column) of the base cell
      double wx, wy;
      if (p < np && dep_cell(a, xp, yp, ix, iy, wx, wy) && iy + 1 >= yb && iy < yb + hb)
        cid = (iy - yb + 1) * bw + (ix - bx0);
      const int lead = __shfl_sync(0xffffffffu, cid, l & ~3);
      const unsigned match = __ballot_sync(0xffffffffu, cid >= 0 && cid == lead);
      const bool same = ((match >> (l & ~3)) & 15u) == 15u;
      // (re, im) of the corners (ix, iy), (ix + 1, iy), (ix, iy + 1), (ix + 1, iy + 1)
      long long c[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      if (cid >= 0) {
        const double q = sqrt(dep_faw2(a, xp, yp)) / gp;
        double sn, cs;
        sincos(hphase * tp, &sn, &cs);
        const double vre = sn * q * scale, vim = cs * q * scale;
        const double w[4] = {wx * wy, (1.0 - wx) * wy, wx * (1.0 - wy), (1.0 - wx) * (1.0 - wy)};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          c[2 * k] = __double2ll_rn(vre * w[k]);
          c[2 * k + 1] = __double2ll_rn(vim * w[k]);
        }
      }
      // a beamlet's sums: lane l ends with the corner of row (l & 2), column (l & 1)
      const bool up = (l & 2) != 0, right = (l & 1) != 0;
      long long k[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        k[i] = (up ? c[4 + i] : c[i]) + __shfl_xor_sync(0xffffffffu, up ? c[i] : c[4 + i], 2);
      const long long cr = (right ? k[2] : k[0]) + __shfl_xor_sync(0xffffffffu, right ? k[0] : k[2], 1);
      const long long ci = (right ? k[3] : k[1]) + __shfl_xor_sync(0xffffffffu, right ? k[1] : k[3], 1);
      if (same) {
        if (up ? cid < ncell : cid >= bw) add((up ? cid : cid - bw) + (right ? 1 : 0), cr, ci);
      } else if (cid >= 0) {
        if (cid >= bw) {
          add(cid - bw, c[0], c[1]);
          add(cid - bw + 1, c[2], c[3]);
        }
        if (cid < ncell) {
          add(cid, c[4], c[5]);
          add(cid + 1, c[6], c[7]);
        }
      }
    }
    __syncthreads();
    double2* out = S + (size_t)(yb - by0) * bw;
    for (int i = tid; i < ncell; i += blockDim.x) {
      const long long sr = (long long)(((unsigned long long)(unsigned int)hre[i] << 32) | lre[i]);
      const long long si = (long long)(((unsigned long long)(unsigned int)him[i] << 32) | lim[i]);
      out[i] = make_double2((double)sr * unscale, (double)si * unscale);
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------- host side ---

static constexpr double kVacimp = 376.73031346177;  // upstream `vacimp`
static constexpr double kEev = 510998.95;          // upstream `eev`

template <typename T, int M, bool PX, int L>
static int configure_pass_t(int device) {
  static std::atomic<uint64_t> configured{0};  // per instantiation, one bit per device
  if (device < 64 && (configured.load() >> device) & 1) return G4B_OK;
  // static + dynamic shared memory must fit the 227 KB a CTA may use
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, adi_pass_kernel<T, M, PX, L>);
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncGetAttributes(adi_pass)");
  e = cudaFuncSetAttribute(adi_pass_kernel<T, M, PX, L>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           227 * 1024 - (int)fa.sharedSizeBytes);
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(adi_pass)");
  if (device < 64) configured.fetch_or(1ull << device);
  return G4B_OK;
}

template <typename T, int M, bool PX, int L>
static int launch_pass_t(g4b_field* f, const AdiPassArgs& args, const void* row,
                         const CUtensorMap& tm, size_t smem) {
  constexpr int W = BandW<T, L>::value;  // warps per CTA
  auto kern = adi_pass_kernel<T, M, PX, L>;
  if (int rc = configure_pass_t<T, M, PX, L>(f->ctx->device)) return rc;
  const unsigned grid = (unsigned)(f->nslice * args.nband);
  {
    LaunchScope ls(f->ctx, PX ? "adi_pass_x" : "adi_pass_y");
    G4B_CUDA_TRY(launch_pdl(kern, grid, W * 32, smem, f->ctx->stream, args,
                            *static_cast<const RowConst<typename CT<T>::type>*>(row), tm));
  }
  return check_launch(f->ctx, "adi_pass_kernel");
}

// Kernel modes: M (odd elements per lane) with 32-lane rows, 100 + M with
// 16-lane rows (FP32 only).
#define G4B_MODES32(X) X(1, 32) X(3, 32) X(5, 32) X(7, 32) X(9, 32) X(11, 32) X(13, 32) \
  X(15, 32) X(17, 32) X(21, 32) X(25, 32) X(33, 32)
#define G4B_MODES16(X) X(5, 16) X(7, 16) X(9, 16) X(11, 16) X(13, 16) X(15, 16) X(17, 16) \
  X(21, 16) X(25, 16) X(33, 16)

template <typename T, bool PX>
static int configure_pass_m(int mode, int device) {
#define G4B_CFG(m, l) \
  case (l == 16 ? 100 : 0) + m: return configure_pass_t<T, m, PX, l>(device);
  if constexpr (sizeof(T) == 8) {
    switch (mode) { G4B_MODES32(G4B_CFG) }
  } else {
    switch (mode) { G4B_MODES32(G4B_CFG) G4B_MODES16(G4B_CFG) }
  }
#undef G4B_CFG
  return fail(G4B_ERR_RANGE, "adi: unsupported elements per lane");
}

int adi_configure(g4b_field* f) {
  const int M = f->mode;
  const int d = f->ctx->device;
  if (f->precision == G4B_FP64) {
    if (int rc = configure_pass_m<double, true>(M, d)) return rc;
    return configure_pass_m<double, false>(M, d);
  }
  if (int rc = configure_pass_m<float, true>(M, d)) return rc;
  return configure_pass_m<float, false>(M, d);
}

template <typename T, bool PX>
static int launch_pass_m(int mode, g4b_field* f, const AdiPassArgs& args, const void* row,
                         const CUtensorMap& tm, size_t smem) {
#define G4B_LAUNCH(m, l) \
  case (l == 16 ? 100 : 0) + m: return launch_pass_t<T, m, PX, l>(f, args, row, tm, smem);
  if constexpr (sizeof(T) == 8) {
    switch (mode) { G4B_MODES32(G4B_LAUNCH) }
  } else {
    switch (mode) { G4B_MODES32(G4B_LAUNCH) G4B_MODES16(G4B_LAUNCH) }
  }
#undef G4B_LAUNCH
  return fail(G4B_ERR_RANGE, "adi: unsupported elements per lane");
}

int adi_plan(g4b_adi* adi, g4b_field* f, const void* src, const int4* desc,
             const AdiYExtras* ex, AdiPlan& P) {
  const int n = f->ngrid, ld = f->ld, W = f->band_rows;
  AdiPassArgs args{};
  args.n = n;
  args.ld = ld;
  args.nband = (n + W - 1) / W;
  args.r = adi->r;
  args.err = f->ctx->d_error;
  args.box_rows = f->store_box_rows;
  args.nbox = f->store_nbox;
  if (f->precision == G4B_FP64) {
    args.tab = adi->d_tab64;
    P.row = &adi->k64;
  } else if (f->mode == adi->mode32) {
    args.tab = adi->d_tab32;
    P.row = &adi->k32;
  } else if (f->mode == adi->mode32_alt && adi->d_tab32_alt) {
    args.tab = adi->d_tab32_alt;
    P.row = &adi->k32_alt;
  } else
    return fail(G4B_ERR_STATE, "adi: solver and field row layouts differ");
  const size_t cb = f->cell_bytes;
  const size_t out_bytes = (size_t)f->store_nbox * f->store_box_rows * W * cb;
  auto smem_for = [&](bool px, bool with_src) {
    size_t tile = (size_t)((px ? W + 2 : W) * ld) * cb;
    if (px && with_src) tile += (size_t)W * ld * cb;
    // pass X: the output staging tile reuses the input tile's memory
    // (written after a barrier that ends every read of the input), which
    // keeps three CTAs of 16-lane rows on an SM; pass Y: after the input
    if (px) {
      args.out_off = 0;
      return std::max(tile, out_bytes);
    }
    const size_t out_off = (tile + 127) / 128 * 128;
    args.out_off = (int)out_off;
    return out_off + out_bytes;
  };
  P.M = f->precision == G4B_FP64 ? adi->M : f->mode;
  if (P.M != f->mode) return fail(G4B_ERR_STATE, "adi: solver and field row layouts differ");
  P.precision = f->precision;
  P.grid = (unsigned)(f->nslice * args.nband);
  P.tm_x = &f->tm_store_b;
  P.tm_y = &f->tm_store_a;
  // pass X: a -> b (transposed R')
  args.in = f->a;
  args.src = src;
  args.desc = desc;
  args.src_cap = (size_t)f->ngrid * f->ld;
  P.smem_x_max = smem_for(true, true);
  P.smem_x = smem_for(true, src != nullptr);
  if (P.smem_x + 2048 > 227 * 1024)
    return fail(G4B_ERR_RANGE, "adi: pass X tile exceeds shared memory");
  P.x = args;
  // pass Y: b -> a (natural)
  args.in = f->b;
  args.src = nullptr;
  args.nslice = f->nslice;
  if (ex) {
    args.zero_start = ex->zero_start;
    args.zero_count = ex->zero_count;
    args.diag = ex->diag;
  }
  P.smem_y = smem_for(false, false);
  P.y = args;
  return G4B_OK;
}

int adi_launch(g4b_field* f, const AdiPlan& P) {
  int rc = P.precision == G4B_FP64
               ? launch_pass_m<double, true>(P.M, f, P.x, P.row, *P.tm_x, P.smem_x)
               : launch_pass_m<float, true>(P.M, f, P.x, P.row, *P.tm_x, P.smem_x);
  if (rc) return rc;
  return P.precision == G4B_FP64
             ? launch_pass_m<double, false>(P.M, f, P.y, P.row, *P.tm_y, P.smem_y)
             : launch_pass_m<float, false>(P.M, f, P.y, P.row, *P.tm_y, P.smem_y);
}

int adi_run(g4b_adi* adi, g4b_field* f, const void* src, const int4* desc,
            const AdiYExtras* ex) {
  AdiPlan P;
  if (int rc = adi_plan(adi, f, src, desc, ex, P)) return rc;
  return adi_launch(f, P);
}

template <int M, bool PX, int L>
static int batch_launch_t(g4b_ctx* c, cudaStream_t st, const AdiBatchArgs& b, size_t smem,
                          int grid) {
  static std::atomic<uint64_t> configured{0};
  auto kern = adi_batch_kernel<float, M, PX, L>;
  if (c->device >= 64 || !((configured.load() >> c->device) & 1)) {
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, kern);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncGetAttributes(adi_batch)");
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             227 * 1024 - (int)fa.sharedSizeBytes);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(adi_batch)");
    if (c->device < 64) configured.fetch_or(1ull << c->device);
  }
  {
    LaunchScope ls(c, PX ? "batch_adi_x" : "batch_adi_y");
    kern<<<grid, BandW<float, L>::value * 32, smem, st>>>(b);
  }
  return check_launch(c, "adi_batch_kernel");
}

int adi_batch_launch(g4b_ctx* c, cudaStream_t st, int mode, bool px, const AdiBatchArgs& b,
                     size_t smem, int grid) {
#define G4B_BATCH_CASE(m, l)                                                   \
  case (l == 16 ? 100 : 0) + m:                                                \
    return px ? batch_launch_t<m, true, l>(c, st, b, smem, grid)               \
              : batch_launch_t<m, false, l>(c, st, b, smem, grid);
  switch (mode) { G4B_MODES32(G4B_BATCH_CASE) G4B_MODES16(G4B_BATCH_CASE) }
#undef G4B_BATCH_CASE
  return fail(G4B_ERR_RANGE, "adi: unsupported elements per lane");
}

// adi_compute_slice_scl + the deterministic deposition
// (src/Core/FieldSolverADICUDA.cpp:75-174) of an FP64 beam into the field's
// compact source tiles; shared by the ADI and FFT solvers.
int fp64_deposit(g4b_field* f, g4b_beam* b, const g4b_step* st, double fc) {
  g4b_ctx* c = f->ctx;
  const int harm = f->harm;
  DepositArgs da{};
  da.x = b->x;
  da.y = b->y;
  da.gamma = b->gamma;
  da.theta = b->theta;
  da.off = b->d_off;
  da.current = b->d_current;
  da.fc = fc;
  da.xks = f->xks;
  da.delz = st->delz;
  da.vacimp = kVacimp;
  da.eev = kEev;
  da.src = static_cast<double2*>(f->src);
  da.desc = f->desc;
  da.src_cap = (size_t)f->ngrid * f->ld;
  da.nslice = f->nslice;
  da.n = f->ngrid;
  da.ld = f->ld;
  da.first = f->first;
  da.harm = harm;
  da.gridmax = f->gridmax;
  da.dgrid = f->dgrid;
  da.ax = st->ax;
  da.ay = st->ay;
  da.kx = st->kx;
  da.ky = st->ky;
  da.gradx = st->gradx;
  da.grady = st->grady;
  da.err = c->d_error;
  const size_t acc_bytes = kDepFp64Acc;
  da.acc_cells = (int)(acc_bytes / 16);
  da.inv_dgrid = 1.0 / f->dgrid;
  G4B_CUDA_TRY(cudaFuncSetAttribute(deposit_slice_kernel,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)acc_bytes));  // per device, cheap
  {
    LaunchScope ls(c, "deposit");
    G4B_CUDA_TRY(launch_pdl(deposit_slice_kernel, (unsigned)f->nslice, kDepFp64Threads,
                            acc_bytes, c->stream, da));
  }
  if (int rc = check_launch(c, "deposit_slice_kernel")) return rc;
  return G4B_OK;
}

}  // namespace g4b

using namespace g4b;

namespace {

using cld = std::complex<long double>;

// Coefficients of rows of n elements held by L lanes of M, rounded to C, and
// their device image: K, then the lanes' wall coefficients.
template <typename C>
void row_tables(double r, int n, int M, int L, RowConst<C>& K, std::vector<unsigned char>& image) {
  using T = decltype(C{}.x);
  const cld ir(0.0L, r), beta = (cld(1.0L, 2.0L * r) + std::sqrt(cld(1.0L, 4.0L * r))) / 2.0L;
  const cld q = ir / beta;
  // products of long doubles by their parts (std::complex's operator tests for
  // NaN), each table by recurrence: at most a few dozen roundings of 2^-64
  auto mul = [](cld a, cld b) {
    return cld(a.real() * b.real() - a.imag() * b.imag(),
               a.real() * b.imag() + a.imag() * b.real());
  };
  auto power = [&](long long m) {  // q^m by squaring
    cld p = 1.0L, s = q;
    for (; m > 0; m >>= 1, s = mul(s, s))
      if (m & 1) p = mul(p, s);
    return p;
  };
  // (what is below half the smallest denormal by a comparison: a conversion
  // that underflows takes 150 ns, most of a table's time)
  constexpr long double tiny = std::numeric_limits<T>::denorm_min() / 4.0L;
  auto round1 = [](long double x) {
    return std::fabs(x) < tiny ? std::copysign((T)0, (T)(x < 0 ? -1 : 1)) : (T)x;
  };
  auto round = [&](cld z) {
    C c;
    c.x = round1(z.real());
    c.y = round1(z.imag());
    return c;
  };
  K = RowConst<C>{};
  cld p = 1.0L, qM = 1.0L;
  for (int m = 0; m < kRowMaxM + 2; ++m, p = mul(p, q)) {
    K.P[m] = round(p);
    if (m == M) qM = p;
  }
  K.cb = round(1.0L / beta);
  // scan steps whose multiplier rounds to zero are left out (no more than that:
  // the field far outside the beam is a power of q, small but exact)
  p = qM;
  for (int t = 0; (1 << t) < L; ++t, p = mul(p, p)) {
    K.A[t] = round(p);
    if (K.A[t].x != 0 || K.A[t].y != 0) K.nscan = t + 1;
  }
  std::vector<C> wall(2 * L, C{0, 0});
  const cld inv = 1.0L / (1.0L - power(2LL * n + 2));
  const int lanes = (n + M - 1) / M;
  p = inv;
  for (int l = 0; l < lanes; ++l, p = mul(p, qM)) wall[l] = round(p);
  p = mul(power(2LL * n + 2 - (long long)lanes * M), inv);
  for (int l = lanes - 1; l >= 0; --l, p = mul(p, qM)) wall[L + l] = round(p);
  image.resize(sizeof K + wall.size() * sizeof(C));
  std::memcpy(image.data(), &K, sizeof K);
  std::memcpy(image.data() + sizeof K, wall.data(), wall.size() * sizeof(C));
}

}  // namespace

extern "C" {

int g4b_adi_create(g4b_ctx* c, g4b_adi** out) {
  if (!c || !out) return fail(G4B_ERR_ARG, "g4b_adi_create: null arg");
  g4b_adi* a = new (std::nothrow) g4b_adi();
  if (!a) return fail(G4B_ERR_NOMEM, "g4b_adi_create: host allocation");
  a->ctx = c;
  ctx_retain(c);
  *out = a;
  return G4B_OK;
}

int g4b_adi_destroy(g4b_adi* a) {
  if (!a) return G4B_OK;
  ctx_quiesce(a->ctx);
  dev_free(a->ctx, a->d_tab64);
  dev_free(a->ctx, a->d_tab32);
  dev_free(a->ctx, a->d_tab32_alt);
  ctx_release(a->ctx);
  delete a;
  return G4B_OK;
}

// FieldSolverADICUDA::init (src/Core/FieldSolverADICUDA.cpp:821-866): the
// coefficients of the row solve, in long double, for every row layout a field
// of this grid may take.
int g4b_adi_init(g4b_adi* a, double delz, double dgrid, double xks, int ngrid) {
  if (!a) return fail(G4B_ERR_ARG, "g4b_adi_init: null adi");
  if (ngrid < 2 || !(dgrid > 0) || !(xks > 0))
    return fail(G4B_ERR_ARG, "g4b_adi_init: bad arguments");
  if (a->ready && delz == a->delz && ngrid == a->ngrid && dgrid == a->dgrid &&
      xks == a->xks)
    return G4B_OK;
  const int M = pick_M(ngrid);
  if (!M) return fail(G4B_ERR_RANGE, "g4b_adi_init: ngrid above 1056 is not supported");
  const int n = ngrid;
  const double r = 0.25 * delz / (xks * dgrid * dgrid);
  g4b_ctx* ctx = a->ctx;
  G4B_CUDA_TRY(cudaSetDevice(ctx->device));
  if (a->d_tab64) {
    cudaStreamSynchronize(ctx->stream);
    for (void** d : {&a->d_tab64, &a->d_tab32, &a->d_tab32_alt}) {
      dev_free(a->ctx, *d);
      *d = nullptr;
    }
    a->ready = false;
  }
  // FP64 fields solve rows with 32 lanes; FP32 fields with the layout of
  // their mode (16-lane rows where those fit the row more closely), or the
  // other FP32 layout, which the batch tuner may pick
  const int mode32 = pick_mode(n, G4B_MIXED), mode32_alt = alt_mode(n);
  std::vector<unsigned char> t64, t32, t32a;
  row_tables(r, n, M, 32, a->k64, t64);
  row_tables(r, n, mode_M(mode32), mode_L(mode32), a->k32, t32);
  if (mode32_alt) row_tables(r, n, mode_M(mode32_alt), mode_L(mode32_alt), a->k32_alt, t32a);
  const std::pair<void**, std::vector<unsigned char>*> up[] = {
      {&a->d_tab64, &t64}, {&a->d_tab32, &t32}, {&a->d_tab32_alt, &t32a}};
  for (auto& [d, t] : up) {
    if (t->empty()) continue;
    G4B_CUDA_TRY(dev_alloc(ctx, d, t->size()));
    G4B_CUDA_TRY(cudaMemcpyAsync(*d, t->data(), t->size(), cudaMemcpyHostToDevice, ctx->stream));
  }
  G4B_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  a->ngrid = ngrid;
  a->delz = delz;
  a->dgrid = dgrid;
  a->xks = xks;
  a->r = r;
  a->M = M;
  a->mode32 = mode32;
  a->mode32_alt = mode32_alt;
  a->ready = true;
  return G4B_OK;
}

// FieldSolverADICUDA::advance (src/Core/FieldSolverADICUDA.cpp:638-818).
int g4b_adi_advance(g4b_adi* adi, g4b_field* f, g4b_beam* b, const g4b_step* st,
                    double fc, int enabled) {
  if (!adi || !f || !b || !st) return fail(G4B_ERR_ARG, "g4b_adi_advance: null arg");
  if (!adi->ready || adi->ngrid != f->ngrid)
    return fail(G4B_ERR_STATE,
                "g4b_adi_advance: called before g4b_adi_init for this ngrid");
  if (b->nslice != f->nslice)
    return fail(G4B_ERR_ARG, "g4b_adi_advance: beam and field slice counts differ");
  if (f->precision != G4B_FP64 || b->precision != G4B_FP64)
    return fail(G4B_ERR_ARG, "g4b_adi_advance: the drop-in path holds FP64 state");
  g4b_ctx* c = f->ctx;
  G4B_CUDA_TRY(cudaSetDevice(c->device));
  const int harm = f->harm;
  const bool do_source = st->in_undulator && enabled && (harm % 2) == 1;
  const bool use_source = do_source && b->npart > 0;
  const void* src = nullptr;
  if (use_source) {
    if (int rc = fp64_deposit(f, b, st, fc)) return rc;
    src = f->src;
  }
  return adi_run(adi, f, src, f->desc, nullptr);
}

}  // extern "C"
