// g4b_fft.cu -- the spectral field solver (FieldSolverFFTCUDA,
// src/Core/FieldSolverFFTCUDA.cpp:157-483) for sm_100a, with its transforms
// written here (no cuFFT).
//
// One field step u' = IFFT2( FFT2(u) exp(i k2 dz) + 2 filter FFT2(S) ) / n^2.
// The phase k2 = -(dx^2 + dy^2) dk^2 / (2 ks) is a sum over the axes, so the
// propagator is a product p(kx) p(ky) and acts on u as one circular
// convolution of length n along x and one along y with the kernel
// c = IDFT_n(p): a convolution per line and axis, where a forward and an
// inverse n-point transform would take two.  The source enters
//   unfiltered : as + 2 S (the inverse transform of 2 S^ is 2 S);
//   filtered   : through its own 2-D transform pair (the sigmoid filter is a
//                function of the radius and does not separate), Bluestein's
//                chirp-z lines: DFT_n(x)_k = w_k (a * h)_k, w_j =
//                exp(-i pi j^2 / n), a_j = x_j w_j, h_t = conj(w_t).
//
//   deposition : the deterministic FP64 source of the ADI solver (compact
//                per-slice tiles; src/Core/FieldSolverFFTCUDA.cpp:77-155 is the
//                same arithmetic as the ADI deposition);
//   unfiltered : rows (convolution along x, in place), columns (along y, in
//                place, + 2 S);
//   filtered   : the source tile's rows forward, its columns forward, times
//                2 filter, back; then u's columns, and u's rows with the
//                source's rows back added.
// A step without a source is the unfiltered pair.
//
// Every line, n <= 256, is one circular convolution of length 512 >= 2n - 1:
// FFT_512, times the precomputed FFT_512 of the kernel, inverse FFT_512.
// A line belongs to 64 threads of eight values each; with j = j0 + 8 j1 +
// 64 j2 and k = k0 + 8 k1 + 64 k2 the FFT is three radix-8 stages (decimation
// in frequency):
//   A: thread t = j0 + 8 j1 over j2 -> k0, times W_512^(t k0); the inputs at
//      and beyond 256 are zeros, so half of its first butterflies drop out;
//   B: thread (k0, j0) = (t / 8, t % 8) over j1 -> k1, times W_64^(j0 k1);
//   C: thread (k0, k1) over j0 -> k2;
// and the inverse runs them back with conjugate twiddles, its last stage for
// the first 256 outputs only.  Between stages the values cross a buffer of
// rows of nine entries (conflict-free 16-byte accesses).  A thread rewrites
// only entries it read itself, so the only barriers are the ones before the
// reads: one over the line's two warps between A and B, a warp's between B
// and C.
//
// Bound: the FP64 pipe (about 530 FP64 instructions per thread and line, half
// an SM clock per warp each) and the exchanges (64 16-byte accesses per thread,
// four clocks per warp each) take about the same time, some 600 clocks per line
// together when overlapped; measured, 1024 slices of 201^2 (CUDA events): rows
// 0.62 ms, columns 0.94 ms, against 1.27 + 2.31 + 1.59 ms for the forward, middle
// and inverse passes of a full transform pair with a line per warp (sixteen
// values per thread, 128 registers); cuFFT's forward and inverse pair takes 4.99
// ms.  The field step with its source: 5.48 -> 1.76 ms.  The order of the spectrum
// (thread t, slot s) -> k = t / 8 + 8 (t % 8) + 64 brev3(s) is seen by the
// pointwise multiply alone.
#include <algorithm>
#include <cmath>
#include <complex>
#include <new>
#include <vector>

#include "g4b_internal.cuh"

namespace g4b {
namespace {

constexpr int kFftM = 512;       // convolution length
constexpr int kFftMaxN = 256;    // 2 n - 1 <= 512
constexpr int kLineT = 64;       // threads per line
constexpr int kTwA = kFftM;              // W_512^(k t), k = 1, 2, 4, t < 64
constexpr int kTwB = kTwA + 3 * kLineT;  // W_64^(k t), k = 1, 2, 4, t < 8
constexpr int kTwAll = kTwB + 3 * 8;
constexpr int kRowLines = 4;     // lines per CTA along x
constexpr int kColLines = 4;     // lines per CTA along y (64-byte row segments)
constexpr int kXbRow = 9;                   // padded row of eight
constexpr int kXb = 8 * 8 * kXbRow;         // exchange buffer of a line (double2)

struct FftArgs {
  const double2* tw;      // W_512^j, j < 512, the lines' factors (kTwA, kTwB), W_512^j's second words
  const double2* chirp;   // w_j, j < n
  const double2* hc;      // FFT_512 of the propagation kernel / 512, slot * 64 + t
  const double2* hf;      // FFT_512(conj w) / 512
  const double2* hi;      // FFT_512(w) / 512
  const double* sig_t;    // source filter, [kx][ky] (filtered runs)
  double2* u;             // field, [slice][iy][ld]
  double2* st;            // source spectrum, [slice][iy or ky][ld] (filtered runs)
  const double2* src;     // compact source tiles
  const int4* desc;       // per-slice tile (x0, y0, width, height)
  size_t src_cap;
  int n, ld, nband;
  double scale;           // 1 / n^2
};

__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 zsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
// a * conj(b)
__device__ __forceinline__ double2 zmulc(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -a.x * b.y));
}
__host__ __device__ constexpr int brev3(int k) { return ((k & 1) << 2) | (k & 2) | ((k & 4) >> 2); }

// t / sqrt2 with sqrt2 / 2 as two words: every transform of every step meets the
// first one's error, always the same way (24 source-free steps at 151^2, a
// Gaussian beam: 8.8e-15 rms without the second, 4.0e-15 with it; 256 slices of
// 201^2: 400 and 413 us).
constexpr double kS = 0.70710678118654752440, kSl = -4.8336466567264565e-17;
__device__ __forceinline__ double by_s(double t) { return fma(kS, t, kSl * t); }

__device__ __forceinline__ double2 mul_w1(double2 z) {  // x (1 - i)/sqrt2
  return make_double2(by_s(z.x + z.y), by_s(z.y - z.x));
}
__device__ __forceinline__ double2 mul_w2(double2 z) { return make_double2(z.y, -z.x); }  // x (-i)
__device__ __forceinline__ double2 mul_w3(double2 z) {  // x (-1 - i)/sqrt2
  return make_double2(by_s(z.y - z.x), by_s(-z.x - z.y));
}
__device__ __forceinline__ double2 mul_c1(double2 z) {  // x (1 + i)/sqrt2
  return make_double2(by_s(z.x - z.y), by_s(z.x + z.y));
}
__device__ __forceinline__ double2 mul_c2(double2 z) { return make_double2(-z.y, z.x); }  // x i
__device__ __forceinline__ double2 mul_c3(double2 z) {  // x (-1 + i)/sqrt2
  return make_double2(by_s(-z.x - z.y), by_s(z.x - z.y));
}

// 8-point DFT of v[0..7] (radix-2, decimation in frequency): X[k] lands in
// slot brev3(k).  HALF: v[4..7] are taken as zeros.
template <bool HALF>
__device__ __forceinline__ void dft8(double2 (&v)[8]) {
  if (HALF) {
    v[4] = v[0];
    v[5] = mul_w1(v[1]);
    v[6] = mul_w2(v[2]);
    v[7] = mul_w3(v[3]);
  } else {
    double2 x = v[0], y = v[4];
    v[0] = zadd(x, y);
    v[4] = zsub(x, y);
    x = v[1], y = v[5];
    v[1] = zadd(x, y);
    v[5] = mul_w1(zsub(x, y));
    x = v[2], y = v[6];
    v[2] = zadd(x, y);
    v[6] = mul_w2(zsub(x, y));
    x = v[3], y = v[7];
    v[3] = zadd(x, y);
    v[7] = mul_w3(zsub(x, y));
  }
#pragma unroll
  for (int blk = 0; blk < 8; blk += 4) {
    double2 x = v[blk], y = v[blk + 2];
    v[blk] = zadd(x, y);
    v[blk + 2] = zsub(x, y);
    x = v[blk + 1], y = v[blk + 3];
    v[blk + 1] = zadd(x, y);
    v[blk + 3] = mul_w2(zsub(x, y));
  }
#pragma unroll
  for (int blk = 0; blk < 8; blk += 2) {
    const double2 x = v[blk], y = v[blk + 1];
    v[blk] = zadd(x, y);
    v[blk + 1] = zsub(x, y);
  }
}

// Unnormalised inverse of dft8 (decimation in time, conjugate twiddles):
// input in its output order, x[j] in slot j.  HALF: x[0..3] only.
template <bool HALF>
__device__ __forceinline__ void idft8(double2 (&v)[8]) {
#pragma unroll
  for (int blk = 0; blk < 8; blk += 2) {
    const double2 x = v[blk], y = v[blk + 1];
    v[blk] = zadd(x, y);
    v[blk + 1] = zsub(x, y);
  }
#pragma unroll
  for (int blk = 0; blk < 8; blk += 4) {
    double2 x = v[blk], y = v[blk + 2];
    v[blk] = zadd(x, y);
    v[blk + 2] = zsub(x, y);
    x = v[blk + 1], y = mul_c2(v[blk + 3]);
    v[blk + 1] = zadd(x, y);
    v[blk + 3] = zsub(x, y);
  }
  const double2 y[4] = {v[4], mul_c1(v[5]), mul_c2(v[6]), mul_c3(v[7])};
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const double2 x = v[s];
    v[s] = zadd(x, y[s]);
    if (!HALF) v[s + 4] = zsub(x, y[s]);
  }
}

// Slot s holds k = brev3(s): times w^k (CONJ: its conjugate).  w, w^2 and w^4
// are table entries, the others products of them: every step repeats a factor's
// error, and with all powers from w alone, up to seven times its own, they were
// most of what the solver lost over a run (24 source-free steps at 101^2, a
// Gaussian beam: 2.0e-14 rms against 7.5e-15, and 5.0e-15 with every power from
// the table).  256 slices of 201^2: 409 us with one entry, 400 with three, 437
// with seven.
template <bool CONJ>
__device__ __forceinline__ double2 tmul(double2 z, double2 w) { return CONJ ? zmulc(z, w) : zmul(z, w); }
template <bool CONJ, int STRIDE>
__device__ __forceinline__ void twiddle8(double2 (&v)[8], const double2* w) {
  const double2 w1 = __ldg(w), w2 = __ldg(w + STRIDE), w4 = __ldg(w + 2 * STRIDE);
  v[brev3(1)] = tmul<CONJ>(v[brev3(1)], w1);
  v[brev3(2)] = tmul<CONJ>(v[brev3(2)], w2);
  v[brev3(4)] = tmul<CONJ>(v[brev3(4)], w4);
  const double2 w3 = zmul(w2, w1);
  v[brev3(3)] = tmul<CONJ>(v[brev3(3)], w3);
  v[brev3(7)] = tmul<CONJ>(v[brev3(7)], zmul(w4, w3));
  v[brev3(5)] = tmul<CONJ>(v[brev3(5)], zmul(w4, w1));
  v[brev3(6)] = tmul<CONJ>(v[brev3(6)], zmul(w4, w2));
}

// The 64 threads of a line within a CTA.
struct Line {
  int t;             // thread of the line
  int bar;           // named barrier of its two warps
  double2* xb;       // its exchange buffer
  const double2 *wa, *wb;  // powers of W_512^t and of W_64^(t % 8)
  __device__ __forceinline__ void sync() const {
    asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(kLineT) : "memory");
  }
};
__device__ __forceinline__ Line make_line(const FftArgs& a, int line, double2* xall) {
  Line L;
  L.t = threadIdx.x & (kLineT - 1);
  L.bar = 1 + line;
  L.xb = xall + line * kXb;
  L.wa = a.tw + kTwA + L.t;
  L.wb = a.tw + kTwB + (L.t & 7);
  return L;
}

// Circular convolution of length 512 of x[t + 64 r] = v[r], r < 4 (zeros
// beyond), with the kernel of spectrum H; returns the first 256 outputs in
// v[0..3] the same way.  H by plain loads: the propagation spectrum may be
// the preceding kernel's output.
__device__ __forceinline__ void conv512(double2 (&v)[8], const Line& L, const double2* H) {
  const int lo = L.t & 7, hi = L.t >> 3;
  double2* own = L.xb + hi * kXbRow + lo;         // entry (0, j1, j0), k0 rows of 72 apart
  double2* grp = L.xb + hi * 8 * kXbRow + lo;     // entry (k0, 0, j0)
  double2* row = L.xb + hi * 8 * kXbRow + lo * kXbRow;  // entry (k0, k1, 0)
  dft8<true>(v);
  twiddle8<false, kLineT>(v, L.wa);
#pragma unroll
  for (int s = 0; s < 8; ++s) own[brev3(s) * 8 * kXbRow] = v[s];
  L.sync();
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = grp[j * kXbRow];
  dft8<false>(v);
  twiddle8<false, 8>(v, L.wb);
#pragma unroll
  for (int s = 0; s < 8; ++s) grp[brev3(s) * kXbRow] = v[s];
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = row[j];
  dft8<false>(v);
#pragma unroll
  for (int s = 0; s < 8; ++s) v[s] = zmul(v[s], H[s * kLineT + L.t]);
  idft8<false>(v);
#pragma unroll
  for (int j = 0; j < 8; ++j) row[j] = v[j];
  __syncwarp();
#pragma unroll
  for (int s = 0; s < 8; ++s) v[s] = grp[brev3(s) * kXbRow];
  twiddle8<true, 8>(v, L.wb);
  idft8<false>(v);
#pragma unroll
  for (int j = 0; j < 8; ++j) grp[j * kXbRow] = v[j];
  L.sync();
#pragma unroll
  for (int s = 0; s < 8; ++s) v[s] = own[brev3(s) * 8 * kXbRow];
  twiddle8<true, kLineT>(v, L.wa);
  idft8<true>(v);
}

// Rows, four per CTA, two CTAs per SM at up to 128 registers (96 slices of
// 201^2: 65 us; three CTAs at 80 registers 70 us, four at 64 82 us, both with
// spills).  kRowConv: u's rows convolved in place.  kRowSrc: the
// rows of the source tile forward into st (rows outside the tile are zero and
// are neither computed nor stored).  kRowBoth: u's rows convolved, plus the
// rows of st transformed back and scaled.
enum { kRowConv, kRowSrc, kRowBoth };
template <int MODE>
__global__ void __launch_bounds__(kRowLines * kLineT, 2)
    fft_row_kernel(const __grid_constant__ FftArgs a) {
  extern __shared__ __align__(16) double2 sm[];
  ptx::pdl_wait();
  const int n = a.n, s = blockIdx.x / a.nband;
  const int line = threadIdx.x / kLineT;
  const int iy = (blockIdx.x % a.nband) * kRowLines + line;
  if (iy >= n) return;  // whole lines: the barriers are a line's own
  const int4 d = MODE == kRowConv ? make_int4(0, 0, 0, 0) : a.desc[s];
  if (MODE == kRowSrc && (d.z <= 0 || iy < d.y || iy >= d.y + d.w)) return;
  const Line L = make_line(a, line, sm);
  const size_t at = ((size_t)s * n + iy) * a.ld;
  double2 v[8], w[4];
  const bool has_src = MODE != kRowConv && d.z > 0;
  if (has_src) {
    const double2* srow = MODE == kRowSrc ? a.src + (size_t)s * a.src_cap + (size_t)(iy - d.y) * d.z
                                          : a.st + at;
    const int lo = MODE == kRowSrc ? d.x : 0, hi = MODE == kRowSrc ? min(d.x + d.z, n) : n;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = L.t + kLineT * r;
      v[r] = make_double2(0.0, 0.0);
      if (i >= lo && i < hi) {
        const double2 c = __ldg(a.chirp + i);
        v[r] = MODE == kRowSrc ? zmul(srow[i - lo], c) : zmulc(srow[i], c);
      }
    }
    conv512(v, L, MODE == kRowSrc ? a.hf : a.hi);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = L.t + kLineT * r;
      if (i < n) {
        const double2 c = __ldg(a.chirp + i);
        if (MODE == kRowSrc) {
          a.st[at + i] = zmul(v[r], c);
        } else {
          w[r] = zmulc(v[r], c);
          w[r] = make_double2(w[r].x * a.scale, w[r].y * a.scale);
        }
      }
    }
  }
  if constexpr (MODE != kRowSrc) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = L.t + kLineT * r;
      v[r] = i < n ? a.u[at + i] : make_double2(0.0, 0.0);
    }
    conv512(v, L, a.hc);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = L.t + kLineT * r;
      if (i < n) a.u[at + i] = has_src ? zadd(v[r], w[r]) : v[r];
    }
  }
}

// Columns, four per CTA, through a shared tile of the plane's rows (64-byte
// segments in global memory; entry (row, c) of the tile at row * 4 +
// (c ^ row / 2 % 4), so that the threads of a line read its rows without bank
// conflicts).  Three CTAs per SM, 80 registers with 64-84 bytes of spills (96
// slices of 201^2: 94 us with the tile copied by cp.async, 101 us through
// registers; eight columns per CTA 107 us at one and 130 us at two CTAs per SM);
// the two transforms of kColSrc at two (124 against 132 us for 64 slices of
// 255^2).  kColConv: u's columns convolved in place; kColAdd: + 2 S; kColSrc: the
// columns of st forward, times 2 filter, back, in place.
enum { kColConv, kColAdd, kColSrc };
__device__ __forceinline__ int col_swz(int y) { return (y >> 1) & 3; }
template <int MODE>
__global__ void __launch_bounds__(kColLines * kLineT, MODE == kColSrc ? 2 : 3)
    fft_col_kernel(const __grid_constant__ FftArgs a) {
  extern __shared__ __align__(16) double2 sm[];
  ptx::pdl_wait();
  const int n = a.n, s = blockIdx.x / a.nband;
  const int x0 = (blockIdx.x % a.nband) * kColLines, cols = min(kColLines, n - x0);
  const int line = threadIdx.x / kLineT;
  const int4 d = MODE == kColConv ? make_int4(0, 0, 0, 0) : a.desc[s];
  if (MODE == kColSrc && d.z <= 0) return;
  double2* tile = sm + kColLines * kXb;
  double2* plane = (MODE == kColSrc ? a.st : a.u) + (size_t)s * n * a.ld + x0;
  const int ylo = MODE == kColSrc ? d.y : 0, yhi = MODE == kColSrc ? min(d.y + d.w, n) : n;
  for (int i = threadIdx.x; i < n * kColLines; i += kColLines * kLineT) {
    const int y = i / kColLines, c = i % kColLines;
    double2* to = tile + (i - c + (c ^ col_swz(y)));
    const bool in = c < cols && y >= ylo && y < yhi;
    const double2* from = plane + (in ? (size_t)y * a.ld + c : 0);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ptx::smem_u32(to)), "l"(from),
                 "r"(in ? 16 : 0)
                 : "memory");  // zero-filled outside
  }
  const Line L = make_line(a, line, sm);
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  double2 v[8];
  auto entry = [&](int y) -> double2& { return tile[y * kColLines + (line ^ col_swz(y))]; };
  if (line < cols) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = L.t + kLineT * r;
      v[r] = make_double2(0.0, 0.0);
      if (i < n) v[r] = MODE == kColSrc ? zmul(entry(i), __ldg(a.chirp + i)) : entry(i);
    }
    conv512(v, L, MODE == kColSrc ? a.hf : a.hc);
    if (MODE == kColSrc) {
      // the forward transform's closing chirp w_k and the inverse's opening
      // conj(w_k) cancel (|w_k| = 1)
      const double* sg = a.sig_t + (size_t)(x0 + line) * n;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int k = L.t + kLineT * r;
        const double f = k < n ? 2.0 * __ldg(sg + k) : 0.0;
        v[r] = k < n ? make_double2(v[r].x * f, v[r].y * f) : make_double2(0.0, 0.0);
      }
      conv512(v, L, a.hi);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = L.t + kLineT * r;
      if (i < n) entry(i) = MODE == kColSrc ? zmulc(v[r], __ldg(a.chirp + i)) : v[r];
    }
  }
  __syncthreads();
  const double2* stile = MODE == kColAdd ? a.src + (size_t)s * a.src_cap : nullptr;
  for (int i = threadIdx.x; i < n * kColLines; i += kColLines * kLineT) {
    const int y = i / kColLines, c = i % kColLines;
    if (c >= cols) continue;
    double2 o = tile[i - c + (c ^ col_swz(y))];
    if (MODE == kColAdd) {
      const int sx = x0 + c - d.x, sy = y - d.y;
      if (sx >= 0 && sx < d.z && sy >= 0 && sy < d.w) {
        const double2 sv = stile[(size_t)sy * d.z + sx];
        o = make_double2(fma(2.0, sv.x, o.x), fma(2.0, sv.y, o.y));
      }
    }
    plane[(size_t)y * a.ld + c] = o;
  }
}

// The propagation kernel for a step length and its spectrum: c_t = (1/n) sum_k
// exp(i k1_k dz) exp(2 pi i k t / n) with the one-axis phases k1 (FP64 cos and
// sin as the reference's propagator kernel, src/Core/FieldSolverFFTCUDA.cpp:
// 157-188), then, laid out as h_m = c_m, h_(512-m) = c_(n-m), its 512-point
// transform / 512.  Every step repeats this table's errors, so the roots of unity
// and c carry a second word, products their rounding error, and the sums are
// compensated: beyond the phases' own rounding the spectrum is rounded once.  A
// warp per sum and a launch each: a CTA that forms all of c itself takes n^2 terms.
// 201^2, per change of step length: 20 us in one launch, now 10 (a cluster of
// eight CTAs that exchange c 16; the propagator table of a full transform pair,
// n^2 cosines and sines, 4, in front of field steps of twice the time).
constexpr int kKernThreads = 256, kKernWarps = kKernThreads / 32;
struct CSum {
  double s = 0.0, c = 0.0;
  // + (a + al) (b + bl)
  __device__ __forceinline__ void add(double a, double al, double b, double bl) {
    const double p = a * b;
    c += fma(a, bl, fma(al, b, fma(a, b, -p)));
    ptx::csum_add(s, c, p);
  }
  // The lanes' total, rounded to the first word with the rest in the second.
  __device__ __forceinline__ void total() {
    ptx::csum_warp(s, c, 32);
    const double t = s + c;
    c -= t - s;
    s = t;
  }
  // ... divided by n.
  __device__ __forceinline__ void divide(double n) {
    const double q = s / n;
    c = (fma(-q, n, s) + c) / n;
    s = q;
  }
};
__global__ void __launch_bounds__(kKernThreads)
    fft_kernel_taps(const double* k1, const double2* wn, double delz, int n, double2* taps) {
  __shared__ double2 p[kFftMaxN];
  const int tid = threadIdx.x, lane = tid & 31;
  ptx::pdl_wait();
  if (tid < n) {
    const double ph = k1[tid] * delz;
    p[tid] = make_double2(cos(ph), sin(ph));
  }
  __syncthreads();
  const int t = blockIdx.x * kKernWarps + tid / 32;
  if (t >= n) return;
  CSum re, im;
  for (int k = lane; k < n; k += 32) {
    const double2 w = __ldg(wn + k * t % n), wl = __ldg(wn + n + k * t % n);
    re.add(p[k].x, 0.0, w.x, wl.x);
    re.add(-p[k].y, 0.0, w.y, wl.y);
    im.add(p[k].x, 0.0, w.y, wl.y);
    im.add(p[k].y, 0.0, w.x, wl.x);
  }
  re.total();
  im.total();
  if (lane == 0) {
    re.divide((double)n);
    im.divide((double)n);
    taps[t] = make_double2(re.s, im.s);
    taps[n + t] = make_double2(re.c, im.c);
  }
}
__global__ void __launch_bounds__(kKernThreads)
    fft_kernel_spectrum(const double2* taps, const double2* tw, int n, double2* hc) {
  const int lane = threadIdx.x & 31;
  ptx::pdl_wait();
  const int out = blockIdx.x * kKernWarps + threadIdx.x / 32;
  const int t = out & (kLineT - 1), s = out / kLineT;
  const int k = (t >> 3) + 8 * (t & 7) + 64 * brev3(s);
  CSum re, im;
  for (int m = lane; m < n; m += 32) {
    const double2 e = __ldg(tw + ((k * m) & (kFftM - 1)));
    const double2 el = __ldg(tw + kTwAll + ((k * m) & (kFftM - 1)));
    double2 v = taps[m], vl = taps[n + m];
    re.add(v.x, vl.x, e.x, el.x);
    re.add(-v.y, -vl.y, e.y, el.y);
    im.add(v.x, vl.x, e.y, el.y);
    im.add(v.y, vl.y, e.x, el.x);
    if (m > 0) {  // h_(512-m): the conjugate factor
      v = taps[n - m], vl = taps[2 * n - m];
      re.add(v.x, vl.x, e.x, el.x);
      re.add(v.y, vl.y, e.y, el.y);
      im.add(-v.x, -vl.x, e.y, el.y);
      im.add(v.y, vl.y, e.x, el.x);
    }
  }
  re.total();
  im.total();
  if (lane == 0) hc[out] = make_double2(re.s / kFftM, im.s / kFftM);
}

}  // namespace
}  // namespace g4b

using namespace g4b;

struct g4b_fft {
  g4b_ctx* ctx = nullptr;
  int ngrid = 0;
  double delz = 0, dgrid = 0, xks = 0, prop_delz = 0;
  double xc = 1, yc = 1, sig = 1;   // FieldSolverFFTCUDA's member defaults
  bool want_filter = false;         // initSourceFilter's request
  bool filter = false;              // in effect (shape valid at init)
  bool ready = false;
  double2 *tw = nullptr, *chirp = nullptr, *hf = nullptr, *hi = nullptr;
  double2 *wn = nullptr, *hc = nullptr;
  double* k1 = nullptr;             // one-axis spectral phase per unit length
  double* sig_t = nullptr;
  double2* st = nullptr;            // source spectrum (filtered runs)
  size_t st_cells = 0;
};

namespace {

using cld = std::complex<long double>;

// FFT_512 of h by the definition, in long double, divided by 512 and stored
// in the line FFT's output order (thread t, slot s at s * 64 + t).
std::vector<double2> permuted_spectrum(const std::vector<cld>& h) {
  const long double pi = 3.141592653589793238462643383279502884L;
  std::vector<cld> H(kFftM);
  for (int k = 0; k < kFftM; ++k) {
    cld acc = 0;
    for (int t = 0; t < kFftM; ++t) {
      if (h[t] == cld(0)) continue;
      const long double ang = -2.0L * pi * (long double)((k * t) % kFftM) / kFftM;
      acc += h[t] * cld(cosl(ang), sinl(ang));
    }
    H[k] = acc / (long double)kFftM;
  }
  std::vector<double2> out(kFftM);
  for (int s = 0; s < 8; ++s)
    for (int t = 0; t < kLineT; ++t) {
      const cld v = H[(t >> 3) + 8 * (t & 7) + 64 * brev3(s)];
      out[s * kLineT + t] = make_double2((double)v.real(), (double)v.imag());
    }
  return out;
}

// A root of unity as two words.
void split(long double re, long double im, double2& hi, double2& lo) {
  hi = make_double2((double)re, (double)im);
  lo = make_double2((double)(re - (long double)hi.x), (double)(im - (long double)hi.y));
}

template <typename T>
int upload(g4b_ctx* c, T** d, const std::vector<T>& h) {
  if (*d) dev_free(c, *d);
  *d = nullptr;
  G4B_CUDA_TRY(dev_alloc(c, (void**)d, h.size() * sizeof(T)));
  G4B_CUDA_TRY(cudaMemcpyAsync(*d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice,
                               c->stream));
  return G4B_OK;
}

int set_smem(const void* fn, size_t bytes) {
  G4B_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)bytes));
  return G4B_OK;
}

}  // namespace

extern "C" {

int g4b_fft_create(g4b_ctx* c, g4b_fft** out) {
  if (!c || !out) return fail(G4B_ERR_ARG, "g4b_fft_create: null arg");
  g4b_fft* s = new (std::nothrow) g4b_fft();
  if (!s) return fail(G4B_ERR_NOMEM, "g4b_fft_create: host allocation");
  s->ctx = c;
  ctx_retain(c);
  *out = s;
  return G4B_OK;
}

int g4b_fft_destroy(g4b_fft* s) {
  if (!s) return G4B_OK;
  g4b_ctx* c = s->ctx;
  cudaSetDevice(c->device);
  for (void* p : {(void*)s->tw, (void*)s->chirp, (void*)s->hf, (void*)s->hi,
                  (void*)s->wn, (void*)s->hc, (void*)s->k1, (void*)s->sig_t, (void*)s->st})
    dev_free(c, p);
  delete s;
  ctx_release(c);
  return G4B_OK;
}

// FieldSolverFFTCUDA::initSourceFilter (src/Core/FieldSolverFFTCUDA.cpp:214-222).
int g4b_fft_init_filter(g4b_fft* s, double xc, double yc, double sig, int filter) {
  if (!s) return fail(G4B_ERR_ARG, "g4b_fft_init_filter: null arg");
  s->xc = xc;
  s->yc = yc;
  s->sig = sig;
  s->want_filter = filter != 0 && sig > 0 && xc > 0 && yc > 0;
  s->ready = false;  // the filter table follows the next init
  return G4B_OK;
}

// FieldSolverFFTCUDA::init (src/Core/FieldSolverFFTCUDA.cpp:246-293): the
// one-axis part -dx^2 dk^2 / (2 ks) of the spectral phase, dk = 2 pi / (n
// dgrid), in FFT index order, and the sigmoid source filter; plus the
// Bluestein tables.
int g4b_fft_init(g4b_fft* s, double delz, double dgrid, double xks, int ngrid) {
  if (!s) return fail(G4B_ERR_ARG, "g4b_fft_init: null arg");
  if (ngrid < 2 || ngrid > kFftMaxN)
    return fail(G4B_ERR_RANGE, "g4b_fft_init: ngrid must be in [2, 256]");
  if (!(dgrid > 0) || !(xks > 0)) return fail(G4B_ERR_ARG, "g4b_fft_init: bad dgrid or xks");
  s->delz = delz;
  g4b_ctx* c = s->ctx;
  G4B_CUDA_TRY(cudaSetDevice(c->device));
  if (!(s->ready && s->ngrid == ngrid && s->dgrid == dgrid && s->xks == xks)) {
    const int n = ngrid;
    const long double pi = 3.141592653589793238462643383279502884L;
    std::vector<double2> tw(kTwAll + kFftM), chirp(n), wn(2 * n);  // second words behind
    for (int j = 0; j < kFftM; ++j) {
      const long double ang = -2.0L * pi * j / kFftM;
      split(cosl(ang), sinl(ang), tw[j], tw[kTwAll + j]);
    }
    for (int i = 0; i < 3; ++i) {
      for (int t = 0; t < kLineT; ++t) tw[kTwA + i * kLineT + t] = tw[t << i];
      for (int t = 0; t < 8; ++t) tw[kTwB + i * 8 + t] = tw[8 * t << i];
    }
    std::vector<cld> hfw(kFftM, 0), hiw(kFftM, 0);
    for (int j = 0; j < n; ++j) {
      const long long q = ((long long)j * j) % (2LL * n);
      const long double ang = -pi * (long double)q / n;
      const cld w(cosl(ang), sinl(ang));
      chirp[j] = make_double2((double)w.real(), (double)w.imag());
      const long double turn = 2.0L * pi * (long double)j / n;
      split(cosl(turn), sinl(turn), wn[j], wn[n + j]);
      hfw[j] = std::conj(w);
      hiw[j] = w;
      if (j > 0) {
        hfw[kFftM - j] = std::conj(w);
        hiw[kFftM - j] = w;
      }
    }
    const std::vector<double2> hf = permuted_spectrum(hfw), hi = permuted_spectrum(hiw);
    // the reference's tables (the filter transposed to [kx][ky])
    const bool shape_ok = s->xc > 0 && s->yc > 0 && s->sig > 0;
    const double dk = 4. * asin(1.) / (static_cast<double>(n) * dgrid);
    const double shift = -0.5 * static_cast<double>(n - 1);
    std::vector<double> k1(n), sig_t((size_t)n * n);
    for (int iy = 0; iy < n; iy++) {
      const double dy = static_cast<double>(iy) + shift;
      k1[(iy + (n + 1) / 2) % n] = -dy * dy * dk * dk / 2. / xks;
      const double y = shape_ok ? dy / static_cast<double>(n) / s->yc : 0.0;
      for (int ix = 0; ix < n; ix++) {
        const double dx = static_cast<double>(ix) + shift;
        const double x = shape_ok ? dx / static_cast<double>(n) / s->xc : 0.0;
        const int iiy = (iy + (n + 1) / 2) % n, iix = (ix + (n + 1) / 2) % n;
        const size_t t = (size_t)iix * n + iiy;  // [kx][ky]
        if (shape_ok) {
          const double r = (sqrt(x * x + y * y) - 1) / s->sig;
          sig_t[t] = 1. / (1 + exp(r));
        } else {
          sig_t[t] = 1.0;
        }
      }
    }
    if (int rc = upload(c, &s->tw, tw)) return rc;
    if (int rc = upload(c, &s->chirp, chirp)) return rc;
    if (int rc = upload(c, &s->hf, hf)) return rc;
    if (int rc = upload(c, &s->hi, hi)) return rc;
    if (int rc = upload(c, &s->wn, wn)) return rc;
    if (int rc = upload(c, &s->k1, k1)) return rc;
    if (int rc = upload(c, &s->sig_t, sig_t)) return rc;
    if (!s->hc)  // the spectrum, then the kernel itself
      G4B_CUDA_TRY(dev_alloc(c, (void**)&s->hc, (kFftM + 2 * kFftMaxN) * sizeof(double2)));
    s->prop_delz = std::nan("");
    s->filter = s->want_filter && shape_ok;
    s->ngrid = n;
    s->dgrid = dgrid;
    s->xks = xks;
    s->ready = true;
  }
  if (!(s->prop_delz == delz)) {
    double2* taps = s->hc + kFftM;
    {
      LaunchScope ls(c, "fft_kernel_taps");
      G4B_CUDA_TRY(launch_pdl(fft_kernel_taps, (unsigned)((s->ngrid + kKernWarps - 1) / kKernWarps),
                              kKernThreads, 0, c->stream, s->k1, s->wn, delz, s->ngrid, taps));
    }
    if (int rc = check_launch(c, "fft_kernel_taps")) return rc;
    {
      LaunchScope ls(c, "fft_kernel_spectrum");
      G4B_CUDA_TRY(launch_pdl(fft_kernel_spectrum, kFftM / kKernWarps, kKernThreads, 0, c->stream,
                              taps, s->tw, s->ngrid, s->hc));
    }
    if (int rc = check_launch(c, "fft_kernel_spectrum")) return rc;
    s->prop_delz = delz;
  }
  return G4B_OK;
}

// FieldSolverFFTCUDA::advance (src/Core/FieldSolverFFTCUDA.cpp:295-483).
int g4b_fft_advance(g4b_fft* s, g4b_field* f, g4b_beam* b, const g4b_step* st, double fc,
                    int enabled) {
  if (!s || !f || !b || !st) return fail(G4B_ERR_ARG, "g4b_fft_advance: null arg");
  if (!s->ready || s->ngrid != f->ngrid)
    return fail(G4B_ERR_STATE, "g4b_fft_advance: called before g4b_fft_init for this ngrid");
  if (b->nslice != f->nslice)
    return fail(G4B_ERR_ARG, "g4b_fft_advance: beam and field slice counts differ");
  if (f->precision != G4B_FP64 || b->precision != G4B_FP64)
    return fail(G4B_ERR_ARG, "g4b_fft_advance: the drop-in path holds FP64 state");
  g4b_ctx* c = f->ctx;
  G4B_CUDA_TRY(cudaSetDevice(c->device));
  const int n = f->ngrid;
  const bool do_source = st->in_undulator && enabled && (f->harm % 2) == 1 && b->npart > 0;
  if (do_source)
    if (int rc = fp64_deposit(f, b, st, fc)) return rc;
  const bool filt = do_source && s->filter;
  if (filt) {
    const size_t need = (size_t)f->nslice * n * f->ld;
    if (s->st_cells < need) {
      dev_free(c, s->st);
      s->st = nullptr;
      s->st_cells = 0;
      G4B_CUDA_TRY(dev_alloc(c, (void**)&s->st, need * sizeof(double2)));
      s->st_cells = need;
    }
  }
  FftArgs a{};
  a.tw = s->tw;
  a.chirp = s->chirp;
  a.hc = s->hc;
  a.hf = s->hf;
  a.hi = s->hi;
  a.sig_t = s->sig_t;
  a.u = static_cast<double2*>(f->a);
  a.st = s->st;
  a.src = static_cast<const double2*>(f->src);
  a.desc = f->desc;
  a.src_cap = (size_t)f->ngrid * f->ld;
  a.n = n;
  a.ld = f->ld;
  a.scale = 1.0 / ((double)n * (double)n);
  auto rows = [&](void (*kern)(FftArgs), const char* name) -> int {
    a.nband = (n + kRowLines - 1) / kRowLines;
    const size_t smem = (size_t)kRowLines * kXb * sizeof(double2);
    if (int rc = set_smem((const void*)kern, smem)) return rc;
    {
      LaunchScope ls(c, name);
      G4B_CUDA_TRY(launch_pdl(kern, (unsigned)(f->nslice * a.nband), kRowLines * kLineT, smem,
                              c->stream, a));
    }
    return check_launch(c, "fft_row_kernel");
  };
  auto columns = [&](void (*kern)(FftArgs), const char* name) -> int {
    a.nband = (n + kColLines - 1) / kColLines;
    const size_t smem = (size_t)kColLines * (kXb + n) * sizeof(double2);
    if (int rc = set_smem((const void*)kern, smem)) return rc;
    {
      LaunchScope ls(c, name);
      G4B_CUDA_TRY(launch_pdl(kern, (unsigned)(f->nslice * a.nband), kColLines * kLineT, smem,
                              c->stream, a));
    }
    return check_launch(c, "fft_col_kernel");
  };
  if (filt) {
    if (int rc = rows(fft_row_kernel<kRowSrc>, "fft_src_rows")) return rc;
    if (int rc = columns(fft_col_kernel<kColSrc>, "fft_src_cols")) return rc;
    if (int rc = columns(fft_col_kernel<kColConv>, "fft_cols")) return rc;
    return rows(fft_row_kernel<kRowBoth>, "fft_rows");
  }
  if (int rc = rows(fft_row_kernel<kRowConv>, "fft_rows")) return rc;
  return columns(do_source ? fft_col_kernel<kColAdd> : fft_col_kernel<kColConv>, "fft_cols");
}

}  // extern "C"
