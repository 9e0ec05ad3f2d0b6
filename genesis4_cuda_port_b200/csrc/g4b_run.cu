// g4b_run.cu -- the fused mixed-precision form: a whole FEL run resident on
// the device, advanced by a fixed sequence of kernels per step that a CUDA
// graph replays.
//
// Device state (per particle 28 bytes): x,y and px,py as float2 pairs, the
// energy as an FP32 offset dg = gamma - gamma_ref (keeps the ~0.01 per-step
// energy changes above FP32 resolution), the ponderomotive phase theta in
// FP64.  Fields are complex64.  Per step:
//   K1 beam_step : transverse half step (+chicane), RK4 push with the frozen
//                  bilinear field sample, R56, transverse half step
//                  (+corrector), and each slice's bounding box of touched
//                  cells (integer atomics, order independent);
//   K2 deposit : per slice, the deterministic exact-integer deposition of
//                  every field's source into a compact tile, and the beam
//                  diagnostics (FP64 sums) into the history buffer: a branch of
//                  the captured graph or a kernel beside the deposition in
//                  runs of many slices, CTAs of the same launch in smaller ones;
//   K3/K4 ADI passes per field (pass Y also zeroes the planes this step's
//                  slippage zeroes and writes field-diagnostic partials);
//   K5 diag_finalize : per-slice field diagnostics into the history buffer;
//                  resets the slices' boxes.
// The theta derivative ks(1-1/b) + ku is evaluated cancellation-free in FP64
// as ku - ks*eps/(b(1+b)), eps = btper0/gamma^2 (the two ~ku terms cancel to
// the detuning).  Slippage is the host's integer index model: `first` and the
// zeroed planes of every step are known before the step is enqueued.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <new>
#include <tuple>
#include <vector>

#include "g4b_internal.cuh"

namespace g4b {

constexpr int kRunFields = 8;
constexpr int kStepThreads = 128;  // beam step: two particles per thread
constexpr int kStepBlocks = 8;     // resident beam-step CTAs per SM (<= 64 registers)
constexpr int kStepWarps = kStepThreads / 32;
constexpr int kMaxBunch = 8;
constexpr int kRunMaxNp = 65536;   // particles per slice (deposition scale)
constexpr int kBeamRec = 23;  // reference stats order (DiagnosticCUDA.cpp:102-125)

struct MixField {
  const float2* cells;
  int first, n, ld, nslice, harm, do_source;
  float gridmax, dgrid, inv_dgrid;
  float rtmp;      // fc / xks_h
  int4* bbox;      // [nslice]: ixmin, iymin, ixmax, iymax
};

struct PlaneMapF {
  int mode;
  float strength, offset;
};

struct BeamStepArgs {
  float2 *xy, *pxy;
  float* dg;
  double* th;
  const int4* chunks;
  const double* eloss;
  MixField f[kRunFields];
  int nfield;
  float gref_f, aw, aw2, ax, ay, kx, ky, gradx, grady, half;
  float zt0;          // -2 / xks (FP32)
  double gref, xks, xku, delz, autophase;
  PlaneMapF xm, ym;
  int pre;            // 1 chicane before the first half step
  float m00, m01, m10, m11, m22, m23, m32, m33;
  int post;           // 1 corrector before the second half step
  float cx, cy;
  int has_r56;
  double r56, r56_off;
  int* err;
};

// Reduce an FP64 angle to [-pi, pi) before FP32 trigonometry (the
// hardware sine / cosine, __sincosf, has an absolute error below 2^-21.4 on
// that interval).
__device__ __forceinline__ float reduce_angle(double a) {
  const double twopi = 6.283185307179586476925287;
  return (float)__fma_rn(-twopi, rint(a * (1.0 / twopi)), a);
}

// cell of the deposit / gather in FP32 (the same arithmetic in K1 and K2)
__device__ __forceinline__ bool cell_f(const MixField& f, float x, float y, int& ix, int& iy,
                                       float& wx, float& wy) {
  const float gm = f.gridmax;
  if (!(x > -gm && x < gm && y > -gm && y < gm)) return false;
  // explicit roundings: every kernel computes the same cell and weights
  const float wxr = __fmul_rn(x + gm, f.inv_dgrid), wyr = __fmul_rn(y + gm, f.inv_dgrid);
  const float fx = floorf(wxr), fy = floorf(wyr);  // integers below 2^24: exact
  ix = (int)fx;
  iy = (int)fy;
  if (ix < 0 || ix >= f.n - 1 || iy < 0 || iy >= f.n - 1) return false;
  wx = 1.0f + fx - wxr;
  wy = 1.0f + fy - wyr;
  return true;
}

// ---------------------------------------------------- packed FP32 pairs --
// The beam step advances two particles per thread, one in each lane of a
// packed FP32 pair: sm_100 executes add, subtract, multiply and fused
// multiply-add on f32x2 register pairs as one instruction, so every FP32
// operation of the push serves both particles.  Each lane rounds like the
// scalar IEEE round-to-nearest operation, so a particle's result does not
// depend on its partner.
struct P2 {
  float2 v;
};
__device__ __forceinline__ P2 pr(float a, float b) { return {make_float2(a, b)}; }
__device__ __forceinline__ P2 bc(float a) { return {make_float2(a, a)}; }
__device__ __forceinline__ float& ln(P2& p, int l) { return l ? p.v.y : p.v.x; }
__device__ __forceinline__ float ln(const P2& p, int l) { return l ? p.v.y : p.v.x; }
__device__ __forceinline__ P2 operator+(P2 a, P2 b) { return {__fadd2_rn(a.v, b.v)}; }
__device__ __forceinline__ P2 operator*(P2 a, P2 b) { return {__fmul2_rn(a.v, b.v)}; }
__device__ __forceinline__ P2 fma2(P2 a, P2 b, P2 c) { return {__ffma2_rn(a.v, b.v, c.v)}; }
__device__ __forceinline__ P2 operator-(P2 a, P2 b) {
  P2 r;
  asm("{\n\t.reg .b64 pa, pb, pc;\n\t"
      "mov.b64 pa, {%2, %3};\n\t"
      "mov.b64 pb, {%4, %5};\n\t"
      "sub.rn.f32x2 pc, pa, pb;\n\t"
      "mov.b64 {%0, %1}, pc;\n\t}"
      : "=f"(r.v.x), "=f"(r.v.y)
      : "f"(a.v.x), "f"(a.v.y), "f"(b.v.x), "f"(b.v.y));
  return r;
}

// Thick-lens map of one plane over `half` (advance_focusing_plane,
// src/Core/TrackBeamCUDA.cpp:27-59) for strength s with k = s/gz and
// w2 = k half^2: a1 = cos w, a2 = sin(w)/sqrt(k), a3 = -k a2 (cosh/sinh for
// k < 0, drift for k = 0).  For |w2| < 1e-2 (every undulator and quadrupole
// step of practical lattices) the functions are their Taylor series in w2,
// a1 = 1 - w2/2 + w2^2/24 - w2^3/720 and a2/half = 1 - w2/6 + w2^2/120 -
// w2^3/5040 (truncation < w2^4/40320 < 3e-13); larger phases use the closed
// forms.  lens_coef is one lane of plane2, rounding for rounding.
__device__ __forceinline__ void lens_coef(float k, float w2, float half, float& a1, float& a2) {
  if (fabsf(w2) < 1e-2f) {
    a1 = __fmaf_rn(w2, __fmaf_rn(w2, __fmaf_rn(w2, -1.0f / 720.0f, 1.0f / 24.0f), -0.5f), 1.0f);
    a2 = __fmul_rn(half, __fmaf_rn(w2, __fmaf_rn(w2, __fmaf_rn(w2, -1.0f / 5040.0f,
                                                                 1.0f / 120.0f),
                                                 -1.0f / 6.0f),
                                   1.0f));
  } else if (k > 0.f) {
    const float foc = sqrtf(k);
    float sn, cs;
    sincosf(foc * half, &sn, &cs);
    a1 = cs;
    a2 = sn / foc;
  } else {
    const float foc = sqrtf(-k);
    a1 = coshf(foc * half);
    a2 = sinhf(foc * half) / foc;
  }
}

// c' = a1 (c - o) + a2 p / gz + o,  p' = a1 p + a3 gz (c - o) with
// a3 gz = -a2 k gz = -a2 s (o: the element's offset).
__device__ __forceinline__ void plane2(const PlaneMapF m, float half, P2& c, P2& p, P2 inv_gz) {
  if (m.mode == 0) {
    c = fma2(p, bc(half) * inv_gz, c);
    return;
  }
  const P2 k = bc(m.strength) * inv_gz;
  const P2 w2 = k * bc(half * half);
  P2 a1, a2;
  if (fmaxf(fabsf(w2.v.x), fabsf(w2.v.y)) < 1e-2f) {
    a1 = fma2(w2, fma2(w2, fma2(w2, bc(-1.0f / 720.0f), bc(1.0f / 24.0f)), bc(-0.5f)), bc(1.0f));
    a2 = bc(half) *
         fma2(w2, fma2(w2, fma2(w2, bc(-1.0f / 5040.0f), bc(1.0f / 120.0f)), bc(-1.0f / 6.0f)),
              bc(1.0f));
  } else {
    lens_coef(k.v.x, w2.v.x, half, a1.v.x, a2.v.x);
    lens_coef(k.v.y, w2.v.y, half, a1.v.y, a2.v.y);
  }
  const P2 o = bc(m.offset);
  const P2 xt = c - o;
  c = fma2(a1, xt, fma2(a2 * inv_gz, p, o));
  p = fma2(a2 * bc(-m.strength), xt, a1 * p);
}

// sin and cos of a small angle (|a| < 0.1: Taylor series to a^5 and a^4,
// truncation below a^7/5040 < 2e-11 and a^6/720 < 1.4e-9, under the FP32
// rounding of the results); larger angles use sincosf.  sincos_small is one
// lane of sincos_small2, rounding for rounding.
__device__ __forceinline__ void sincos_small(float a, float& s, float& c) {
  if (fabsf(a) < 0.1f) {
    const float a2 = __fmul_rn(a, a);
    s = __fmul_rn(a, __fmaf_rn(a2, __fmaf_rn(a2, 1.0f / 120.0f, -1.0f / 6.0f), 1.0f));
    c = __fmaf_rn(a2, __fmaf_rn(a2, 1.0f / 24.0f, -0.5f), 1.0f);
  } else {
    sincosf(a, &s, &c);
  }
}

__device__ __forceinline__ void sincos_small2(P2 a, P2& s, P2& c) {
  if (fmaxf(fabsf(a.v.x), fabsf(a.v.y)) < 0.1f) {
    const P2 a2 = a * a;
    s = a * fma2(a2, fma2(a2, bc(1.0f / 120.0f), bc(-1.0f / 6.0f)), bc(1.0f));
    c = fma2(a2, fma2(a2, bc(1.0f / 24.0f), bc(-0.5f)), bc(1.0f));
  } else {
    sincos_small(a.v.x, s.v.x, c.v.x);
    sincos_small(a.v.y, s.v.y, c.v.y);
  }
}

// NF: number of fields when known at compile time (1, 2), 0 = up to 8.
// One CTA of kStepThreads threads advances a chunk of up to 2 kStepThreads
// particles of one slice: thread t holds particles t (lane x) and
// t + kStepThreads (lane y) of the chunk; a dead y lane repeats x and is
// not stored.
template <int NF>
__device__ __forceinline__ void beam_chunk(const BeamStepArgs& a, const int4 ch) {
  constexpr int kF = NF > 0 ? NF : kRunFields;
  const int nfield = NF > 0 ? NF : a.nfield;
  __shared__ int sbb[kRunFields][4][kStepWarps];
  const int slice = ch.x;
  const int tid = threadIdx.x;
  const bool live = tid < ch.z, live_y = tid + kStepThreads < ch.z;
  const int64_t ipx = (((int64_t)ch.w) << 31) + (int64_t)(unsigned)ch.y + tid;
  const int64_t ipy = live_y ? ipx + kStepThreads : ipx;
  int bb[kF][4];
#pragma unroll
  for (int f = 0; f < kF; ++f) {
    bb[f][0] = bb[f][1] = 1 << 30;
    bb[f][2] = bb[f][3] = -1;
  }
  if (live) {
    const float2 xy0 = a.xy[ipx], xy1 = a.xy[ipy], pp0 = a.pxy[ipx], pp1 = a.pxy[ipy];
    P2 x = pr(xy0.x, xy1.x), y = pr(xy0.y, xy1.y), px = pr(pp0.x, pp1.x), py = pr(pp0.y, pp1.y);
    P2 d = pr(a.dg[ipx], a.dg[ipy]);
    double t[2] = {a.th[ipx], a.th[ipy]};
    // TrackBeamCUDA::track, first half (src/Core/TrackBeamCUDA.cpp:156-204)
    {
      if (a.pre) {
#pragma unroll
        for (int l = 0; l < 2; ++l) {
          float &xl = ln(x, l), &pxl = ln(px, l), &yl = ln(y, l), &pyl = ln(py, l);
          const float g = a.gref_f + ln(d, l);
          const float gz = sqrtf(g * g - 1.0f - pxl * pxl - pyl * pyl);
          float tmp = xl;
          xl = a.m00 * tmp + a.m01 * pxl / gz;
          pxl = a.m10 * tmp * gz + a.m11 * pxl;
          tmp = yl;
          yl = a.m22 * tmp + a.m23 * pyl / gz;
          pyl = a.m32 * tmp * gz + a.m33 * pyl;
        }
      }
      const P2 g = bc(a.gref_f) + d;
      const P2 gz2 = fma2(g, g, bc(-1.0f - a.aw2)) - fma2(px, px, py * py);
      const P2 inv_gz = pr(rsqrtf(gz2.v.x), rsqrtf(gz2.v.y));
      plane2(a.xm, a.half, x, px, inv_gz);
      plane2(a.ym, a.half, y, py, inv_gz);
    }
    // BeamSolverCUDA::advance push (src/Core/BeamSolverCUDA.cpp:226-409)
    t[0] += a.autophase;
    t[1] += a.autophase;
    const P2 dxu = x - bc(a.ax), dyu = y - bc(a.ay);
    const P2 awloc =
        fma2(bc(a.gradx), dxu,
             fma2(bc(a.grady), dyu,
                  fma2(bc(0.5f), fma2(bc(a.kx) * dxu, dxu, bc(a.ky) * dyu * dyu), bc(1.0f))));
    const P2 btpar = fma2(bc(a.aw2), awloc * awloc, fma2(py, py, fma2(px, px, bc(1.0f))));
    const float ez = (float)a.eloss[slice];
    // Field sample of each field rotated to the start phase,
    // w = sc (re - i im) e^{-i h theta0} with sc = rtmp awloc: the field term
    // of a stage at phase offset dth is then w e^{-i h dth}.
    P2 wr[kF], wi[kF];
#pragma unroll
    for (int f = 0; f < kF; ++f) {
      wr[f] = wi[f] = bc(0.f);
      if (f >= nfield) continue;
      const MixField& F = a.f[f];
      int islice = slice + F.first;  // both in [0, nslice)
      if (islice >= F.nslice) islice -= F.nslice;
      const float2* base = F.cells + (size_t)islice * F.n * F.ld;
      P2 cre = bc(0.f), cim = bc(0.f), cs0, sn0;
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        int ix, iy;
        float wx, wy;
        if (cell_f(F, ln(x, l), ln(y, l), ix, iy, wx, wy)) {
          const float2* c = base + (size_t)iy * F.ld + ix;
          const float2 c00 = __ldg(c), c10 = __ldg(c + 1), c01 = __ldg(c + F.ld),
                       c11 = __ldg(c + F.ld + 1);
          const float w00 = wx * wy, w10 = (1.f - wx) * wy, w01 = wx * (1.f - wy),
                      w11 = (1.f - wx) * (1.f - wy);
          ln(cre, l) = c00.x * w00 + c10.x * w10 + c01.x * w01 + c11.x * w11;
          ln(cim, l) = c00.y * w00 + c10.y * w10 + c01.y * w01 + c11.y * w11;
        }
        __sincosf(reduce_angle((double)F.harm * t[l]), &ln(sn0, l), &ln(cs0, l));
      }
      wr[f] = (bc(F.rtmp) * awloc) * (cre * cs0 - cim * sn0);
      wi[f] = (bc(-F.rtmp) * awloc) * fma2(cre, sn0, cim * cs0);
    }
    // theta' = ks (1 - 1/b0) + ku with b0 = sqrt(1 - eps), eps = btper0 /
    // gamma^2 ~ 1e-8: the two ~ku terms cancel to the detuning, so the
    // zero-field, start-of-step value A0 = ku - ks eps0 fe(eps0) (fe =
    // 1/(b(1+b))) is formed once in FP64.  Within the step eps differs from
    // eps0 by the relative amount r = (1 + delta/btpar) (g0/gs)^2 - 1, where
    // delta = -(2/ks) Re(c) is the field term (~1e-10 .. 1e-4 of btpar) and
    // gs the stage energy; then ks eps fe(eps) = B0 (1 + r) (1 + O(eps0 r))
    // with B0 = ks eps0 fe(eps0), so theta' = A0 - B0 r to a relative
    // 1e-8 of the field term, and r is formed in FP32 without cancellation.
    // The energy derivative Im(c) / (b0 gs) - ez drops b0 = 1 + O(1e-8).
    P2 A0, nB0, ig0;
#pragma unroll
    for (int l = 0; l < 2; ++l) {
      const double g0 = a.gref + (double)ln(d, l);
      // 1/g0: one Newton step from the FP32 reciprocal (relative error
      // ~2^-44, far below what the FP32 results keep)
      double inv_g0 = (double)__fdividef(1.0f, (float)g0);
      inv_g0 = fma(inv_g0, fma(-g0, inv_g0, 1.0), inv_g0);
      const double eps0 = (double)ln(btpar, l) * inv_g0 * inv_g0;
      const double fe0 = 0.5 + eps0 * (0.375 + eps0 * 0.3125);
      const double B0d = a.xks * eps0 * fe0;
      ln(A0, l) = (float)(a.xku - B0d);
      ln(nB0, l) = -(float)B0d;
      ln(ig0, l) = (float)inv_g0;
    }
    // delta / btpar per unit Re(c)
    const P2 zt = bc(a.zt0) * pr(__fdividef(1.0f, btpar.v.x), __fdividef(1.0f, btpar.v.y));
    const P2 nez = bc(-ez);
    // stage derivatives (energy kg, phase kp) at energy offset ds (from g0)
    // and phase offset dth
    auto ode = [&](P2 ds, P2 dth, P2& kg, P2& kp) {
      P2 ctr = bc(0.f), cti = bc(0.f);
#pragma unroll
      for (int f = 0; f < kF; ++f) {
        if (f >= nfield) break;
        P2 sd, cd;
        sincos_small2(bc((float)a.f[f].harm) * dth, sd, cd);
        if (f == 0) {
          ctr = fma2(wr[0], cd, wi[0] * sd);
          cti = wi[0] * cd - wr[0] * sd;
        } else {
          ctr = fma2(wr[f], cd, fma2(wi[f], sd, ctr));
          cti = fma2(wi[f], cd, cti) - wr[f] * sd;
        }
      }
      const P2 e = ds * ig0;               // (gs - g0) / g0, |e| <~ 1e-3
      const P2 bq = e * (e - bc(1.0f));    // g0 / gs - 1, error O(e^3)
      const P2 ar = zt * ctr;              // delta / btpar
      const P2 r = fma2(bq * (bq + bc(2.0f)), ar + bc(1.0f), ar);
      kp = fma2(nB0, r, A0);
      kg = fma2(cti, fma2(ig0, bq, ig0), nez);
    };
    // Fourth-order Runge-Kutta on the step's energy increment dd and phase
    // increment dt (both small, so FP32 keeps their relative precision; the
    // classical combination that src/Core/BeamSolverCUDA.cpp:258-299 forms
    // in accumulator form); theta and the stored energy offset are updated
    // once at the end
    P2 k1g, k1p;
    {
      // first stage at the start point: no phase rotation, gs = g0
      P2 ctr = wr[0], cti = wi[0];
#pragma unroll
      for (int f = 1; f < kF; ++f) {
        if (f >= nfield) break;
        ctr = ctr + wr[f];
        cti = cti + wi[f];
      }
      k1p = fma2(nB0, zt * ctr, A0);
      k1g = fma2(cti, ig0, nez);
    }
    const P2 hh = bc((float)(0.5 * a.delz)), h = bc((float)a.delz);
    // ug, up: the latest stage's derivatives; sg, sp: k1 + 2 k2 + 2 k3 + k4
    P2 ug, up;
    ode(hh * k1g, hh * k1p, ug, up);
    P2 sg = fma2(bc(2.0f), ug, k1g), sp = fma2(bc(2.0f), up, k1p);
    ode(hh * ug, hh * up, ug, up);
    sg = fma2(bc(2.0f), ug, sg);
    sp = fma2(bc(2.0f), up, sp);
    ode(h * ug, h * up, ug, up);
    const P2 h6 = bc((float)(a.delz / 6.0));
    const P2 dd = h6 * (sg + ug);
    const P2 dt = h6 * (sp + up);
#pragma unroll
    for (int l = 0; l < 2; ++l) {
      t[l] += (double)ln(dt, l);
      ln(d, l) = (float)((double)ln(d, l) + (double)ln(dd, l));
      // applyR56 (src/Core/TrackBeamCUDA.cpp:257-278): theta += R56 (gamma - gamma0)
      if (a.has_r56) t[l] += a.r56 * ((double)ln(d, l) + a.r56_off);
    }
    // second half (+corrector on the last half step)
    {
      if (a.post) {
        px = px + bc(a.cx);
        py = py + bc(a.cy);
      }
      const P2 g = bc(a.gref_f) + d;
      const P2 gz2 = fma2(g, g, bc(-1.0f - a.aw2)) - fma2(px, px, py * py);
      const P2 inv_gz = pr(rsqrtf(gz2.v.x), rsqrtf(gz2.v.y));
      plane2(a.xm, a.half, x, px, inv_gz);
      plane2(a.ym, a.half, y, py, inv_gz);
    }
    a.xy[ipx] = make_float2(x.v.x, y.v.x);
    a.pxy[ipx] = make_float2(px.v.x, py.v.x);
    a.dg[ipx] = d.v.x;
    a.th[ipx] = t[0];
    if (live_y) {
      a.xy[ipy] = make_float2(x.v.y, y.v.y);
      a.pxy[ipy] = make_float2(px.v.y, py.v.y);
      a.dg[ipy] = d.v.y;
      a.th[ipy] = t[1];
    }
#pragma unroll
    for (int f = 0; f < kF; ++f) {
      if (f >= nfield) break;
      if (!a.f[f].do_source) continue;
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        int ix, iy;
        float wx, wy;
        if ((l == 0 || live_y) && cell_f(a.f[f], ln(x, l), ln(y, l), ix, iy, wx, wy)) {
          bb[f][0] = min(bb[f][0], ix);
          bb[f][1] = min(bb[f][1], iy);
          bb[f][2] = max(bb[f][2], ix);
          bb[f][3] = max(bb[f][3], iy);
        }
      }
    }
  }
  // per-CTA bounding boxes -> per-slice (integer min/max: order independent)
  const int w = tid >> 5, l = tid & 31;
#pragma unroll
  for (int f = 0; f < kF; ++f) {
    if (f >= nfield) break;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int v = q < 2 ? __reduce_min_sync(0xffffffffu, bb[f][q])
                          : __reduce_max_sync(0xffffffffu, bb[f][q]);
      if (l == 0) sbb[f][q][w] = v;
    }
  }
  __syncthreads();
  if (tid < 4 * nfield) {
    const int f = tid >> 2, q = tid & 3;
    int v = sbb[f][q][0];
    for (int i = 1; i < kStepWarps; ++i) v = q < 2 ? min(v, sbb[f][q][i]) : max(v, sbb[f][q][i]);
    if (a.f[f].do_source) {
      int* b = reinterpret_cast<int*>(&a.f[f].bbox[slice]) + q;
      if (q < 2) {
        if (v < (1 << 30)) atomicMin(b, v);
      } else if (v >= 0) {
        atomicMax(b, v);
      }
    }
  }
}

template <int NF>
__global__ void __launch_bounds__(kStepThreads, kStepBlocks) beam_step_kernel(const __grid_constant__ BeamStepArgs a) {
  ptx::pdl_wait();
  beam_chunk<NF>(a, a.chunks[blockIdx.x]);
}

// Batched form: items[i] = (run, chunk of that run), per-run arguments.
struct BeamBatchArgs {
  const BeamStepArgs* args;
  const int2* items;
  const int* nitems;
};

template <int NF>
__global__ void __launch_bounds__(kStepThreads, kStepBlocks) beam_batch_kernel(const __grid_constant__ BeamBatchArgs b) {
  const int nitems = *b.nitems;
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const int2 w = b.items[it];
    const BeamStepArgs& a = b.args[w.x];
    beam_chunk<NF>(a, a.chunks[w.y]);
    __syncthreads();
  }
}

// ------------------------------------------------------ deposit + beam diag --
struct DepField {
  float2* src;        // compact tiles, cap cells per slice
  int4* desc;
  int4* bbox;
  int* mpred;         // [nslice] M of the slice's previous deposition (0: none)
  float* qpred;       // [nslice] largest charge weight of the previous deposition (0: none)
  unsigned char* tiles;  // [nslice] DepTile, zero between launches (runs of few slices)
  int tile_cells;
  size_t cap;
  int first, n, ld, nslice, harm, do_source;
  float gridmax, dgrid, inv_dgrid;
  double kscl;        // source scale times particles over current
};

struct DepArgs {
  const float2* xy;
  const float* dg;
  const double* th;
  const int64_t* off;
  const double* current;
  DepField f[kRunFields];
  int nfield;
  float ax, ay, kx, ky, gradx, grady, gref_f;
  double delz;
  int* err;
};

struct BeamDiagArgs {
  const float2 *xy, *pxy;
  const float* dg;
  const double* th;
  const int64_t* off;
  int nbunch, need_aux;
  double gref;
  double* beam_hist;  // [nslice][23 + 2*nbunch] records of this step
};

// Beam diagnostics (DiagnosticCUDA.cpp:102-125): FP64 sums, the minima and
// maxima in FP32 (exact for FP32 state).  The order of the sums is fixed by
// the slice alone, so any number of CTAs gives the same bits: a
// unit of diag_unit_size consecutive particles is summed by one warp (those of a
// lane in order, then the lanes in a tree), unit j belongs to group j mod
// kDiagGroups, a group adds its units in order and the groups are added in a
// tree, both with compensation (csum_*).
constexpr int kDiagThreads = 256;
// Particles of a unit: eight per lane, or with several bunching harmonics, whose
// butterfly of 32 quantities costs as much as three particles, sixteen, in flight
// by fours (no spills then).  By the run's own harmonics, not the kernel's NB: in a
// batch a run of one harmonic shares a kernel with others.  16384 particles per
// slice and eight harmonics, us per step, eight at once / sixteen in fours [one CTA
// per slice with a tree at its end]: 1 slice 43 / 34 [50], 99 107 / 87 [97], 200 170
// / 145 [179]; 1024 particles per warp leave slices of 2048 too few warps.
template <int NB> __device__ __forceinline__ int diag_unit_size(const int nbunch) {
  return NB == 1 || nbunch == 1 ? 256 : 512;
}
constexpr int kDiagGroups = 32;
constexpr int kDiagSums = 12;         // x, x^2, y, y^2, px, px^2, py, py^2, x px, y py, dg, dg^2

// The groups' sums of a slice, in shared memory.
template <int NB>
struct DiagGroups {
  static constexpr int Q = NB <= 2 ? 16 : 32;  // sums, padded: kDiagSums + 2 NB
  double2 sum[kDiagGroups][Q];          // (sum, compensation)
  float ext[kDiagGroups][10];           // per warp: min, max of x, px, y, py, dg
};

// This lane's sum of one unit: quantity lane / (32 / Q).  The lanes are added
// in a butterfly that halves the quantities a lane carries at every level: 15
// exchanges for 16 quantities where a tree per quantity takes 80.  L2: loads past
// L1 (see beam_diag_kernel).
template <int NB, bool L2>
__device__ __forceinline__ double diag_unit(const BeamDiagArgs& a, const float2* xyp,
                                            const float2* pxyp, const float* dgp,
                                            const double* thp, const int np, const int p0,
                                            float (&mn)[5], float (&mx)[5]) {
  constexpr int Q = DiagGroups<NB>::Q;
  const int lane = threadIdx.x & 31;
  constexpr int U = NB <= 2 ? 8 : 4;  // particles in flight per lane
  double v[Q];
#pragma unroll
  for (int k = 0; k < Q; ++k) v[k] = 0.0;
  auto add = [&](const int base) {
    float2 lxy[U], lpp[U];
    float ldg[U];
    double lth[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int p = base + 32 * u + lane;
      if (p < np) {
        lxy[u] = L2 ? __ldcg(xyp + p) : xyp[p];
        lpp[u] = L2 ? __ldcg(pxyp + p) : pxyp[p];
        ldg[u] = L2 ? __ldcg(dgp + p) : dgp[p];
        lth[u] = L2 ? __ldcg(thp + p) : thp[p];
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (base + 32 * u + lane >= np) break;
      const double x = lxy[u].x, y = lxy[u].y, px = lpp[u].x, py = lpp[u].y;
      const double d = ldg[u];
      v[0] += x; v[1] = __fma_rn(x, x, v[1]);
      v[2] += y; v[3] = __fma_rn(y, y, v[3]);
      v[4] += px; v[5] = __fma_rn(px, px, v[5]);
      v[6] += py; v[7] = __fma_rn(py, py, v[7]);
      v[8] = __fma_rn(x, px, v[8]); v[9] = __fma_rn(y, py, v[9]);
      v[10] += d; v[11] = __fma_rn(d, d, v[11]);
      if (a.need_aux) {
        const float f[5] = {lxy[u].x, lpp[u].x, lxy[u].y, lpp[u].y, ldg[u]};
#pragma unroll
        for (int i = 0; i < 5; ++i) {
          mn[i] = fminf(mn[i], f[i]);
          mx[i] = fmaxf(mx[i], f[i]);
        }
      }
      float s1, c1;
      __sincosf(reduce_angle(lth[u]), &s1, &c1);
      float ch = c1, sh = s1;
#pragma unroll
      for (int h = 0; h < NB; ++h) {
        if (h >= a.nbunch) break;
        v[kDiagSums + 2 * h] += ch;
        v[kDiagSums + 2 * h + 1] += sh;
        const float nc = __fmaf_rn(ch, c1, -__fmul_rn(sh, s1));
        const float ns = __fmaf_rn(sh, c1, __fmul_rn(ch, s1));
        ch = nc;
        sh = ns;
      }
    }
  };
  if constexpr (NB == 1) {
    add(p0);
  } else {
#pragma unroll 1
    for (int base = p0; base < min(p0 + diag_unit_size<NB>(a.nbunch), np); base += 32 * U) add(base);
  }
#pragma unroll
  for (int o = 16, h = Q / 2; o > 0; o >>= 1, h >>= 1) {
    if (h > 0) {
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int k = 0; k < Q / 2; ++k) {
        if (k >= h) break;
        const double give = up ? v[k] : v[k + h];
        v[k] = (up ? v[k + h] : v[k]) + __shfl_xor_sync(0xffffffffu, give, o);
      }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
  return v[0];
}

// The groups of slice bs by warp w of nw.
template <int NB, bool L2 = false>
__device__ __forceinline__ void diag_groups(const BeamDiagArgs& a, const int bs, const int w,
                                            const int nw, DiagGroups<NB>& G) {
  constexpr int Q = DiagGroups<NB>::Q;
  const int lane = threadIdx.x & 31;
  const int64_t p0 = a.off[bs];
  const int np = (int)(a.off[bs + 1] - p0);  // at most kRunMaxNp per slice
  const int unit = diag_unit_size<NB>(a.nbunch);
  // minima / maxima of x, px, y, py (reference start values -+1e5) and dg
  float mn[5] = {1.0e5f, 1.0e5f, 1.0e5f, 1.0e5f, INFINITY};
  float mx[5] = {-1.0e5f, -1.0e5f, -1.0e5f, -1.0e5f, -INFINITY};
  for (int g = w; g < kDiagGroups; g += nw) {
    double s = 0.0, c = 0.0;
    for (int u0 = g * unit; u0 < np; u0 += kDiagGroups * unit)
      ptx::csum_add(s, c, diag_unit<NB, L2>(a, a.xy + p0, a.pxy + p0, a.dg + p0, a.th + p0, np, u0,
                                        mn, mx));
    if (lane % (32 / Q) == 0) G.sum[g][lane / (32 / Q)] = make_double2(s, c);
  }
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    float lo = mn[i], hi = mx[i];
    for (int o = 16; o > 0; o >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (lane == 0) {
      G.ext[w][2 * i] = lo;
      G.ext[w][2 * i + 1] = hi;
    }
  }
}

// The slice's record from the groups' sums and the warps' extremes, by a whole
// CTA of T threads: a warp per quantity, a lane per group.
template <int NB, int T>
__device__ __forceinline__ void diag_record(const BeamDiagArgs& a, const int bs,
                                            const DiagGroups<NB>& G) {
  constexpr int kWarps = T / 32;
  __shared__ double total[kDiagSums + 2 * kMaxBunch];
  __shared__ float bound[10];
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  for (int q = w; q < kDiagSums + 2 * a.nbunch; q += kWarps) {
    double2 t = G.sum[lane][q];
    ptx::csum_warp(t.x, t.y, 32);
    if (lane == 0) total[q] = t.x + t.y;
  }
  for (int q = w; q < 10; q += kWarps) {
    float t = G.ext[lane < kWarps ? lane : 0][q];
    for (int o = 16; o > 0; o >>= 1) {
      const float u = __shfl_xor_sync(0xffffffffu, t, o);
      t = q % 2 == 0 ? fminf(t, u) : fmaxf(t, u);
    }
    if (lane == 0) bound[q] = t;
  }
  __syncthreads();
  const int rec = kBeamRec + 2 * a.nbunch;
  if (tid >= rec) return;
  // record (DiagnosticCUDA.cpp:102-125): [0] sum gamma, [1] sum gamma^2,
  // [2..11] the sums of x .. y py, [12] count, [13..22] minima / maxima of x,
  // px, y, py, gamma (gamma = gref + dg is monotonic in dg), then bunching
  const double N = (double)(a.off[bs + 1] - a.off[bs]);
  double t = N;
  if (tid >= kBeamRec) {
    t = total[kDiagSums + tid - kBeamRec];
  } else if (tid >= 13) {
    t = bound[tid - 13];
    if (tid == 21) t = fmin(1.0e7, a.gref + t);
    if (tid == 22) t = fmax(1.0, a.gref + t);
    if (!a.need_aux) t = 0.0;
  } else if (tid == 0) {
    t = __fma_rn(N, a.gref, total[10]);
  } else if (tid == 1) {
    t = __fma_rn(__dmul_rn(N, a.gref), a.gref,
                 __fma_rn(__dmul_rn(2.0, a.gref), total[10], total[11]));
  } else if (tid != 12) {
    t = total[tid - 2];
  }
  a.beam_hist[(size_t)bs * rec + tid] = t;
}

template <int NB, bool BESIDE>
__global__ void __launch_bounds__(kDiagThreads, 2)
    beam_diag_kernel(const __grid_constant__ BeamDiagArgs a) {
  __shared__ DiagGroups<NB> G;
  // launched beside the deposition (deposit_kernel): the beam step, whose
  // output it reads, is complete, since the deposition waited for it before it
  // let this kernel start; but that wait ordered only the deposition's own
  // reads, so the particles are read from L2 (diag_unit), where the beam step's
  // writes are, and not through an L1 that may hold older lines.  The wait for
  // the deposition at its end makes this kernel's completion imply the
  // deposition's
  if (!BESIDE) ptx::pdl_wait();
  diag_groups<NB, BESIDE>(a, blockIdx.x, threadIdx.x >> 5, kDiagThreads / 32, G);
  __syncthreads();
  diag_record<NB, kDiagThreads>(a, blockIdx.x, G);
  if (BESIDE) ptx::pdl_wait();
}

// Deposition (adi_deposit_source_atomic, FieldSolverADICUDA.cpp:98-174),
// one CTA per slice: a deterministic per-cell reduction in exact integer
// arithmetic.  With M the largest number of contributions any output cell
// receives (the sum of the particle counts of its four base cells) and
// qmax the largest charge weight sqrt(faw2) / gamma, the scale
// S = 2^30 / (M' q') for any M' >= M, q' >= qmax rounds every contribution
// c = rint(S q w (sin h theta, cos h theta)) to an int32 with
// |c| <= 2^30 / M', so no cell sum of 32-bit shared-memory integer atomics
// can overflow (re and im in separate planes, so the 32 lanes of a warp
// spread over the banks).  M' and q' come from the slice's previous
// deposition (M + M/4 + 4 and qmax (1 + 2^-6)): one pass counts the
// particles per base cell, takes qmax and adds the contributions at that
// scale, and the band is redone at the exact scale S = 2^30 / (M qmax) in
// the rare case that the counted M or qmax exceeds its bound.  The first
// deposition after a beam upload counts first.
// Integer addition is associative, so the source does not depend on the
// order in which threads add, and each contribution keeps FP32 resolution
// (2^-24 relative, times at most 1.25 M qmax / (M' q')).  Phases are reduced
// to [-pi, pi) in FP64 and their sine and cosine taken with the hardware
// approximation (absolute error below 2^-21.4 on that interval).  Every
// rounding that could be fused differently is written out with intrinsics,
// so the single-run and the batched kernels give the same bits.  The tile is
// the slice's bounding box of touched cells (from K1); larger tiles
// are processed in row bands.
//
// A slice belongs to one CTA, which holds a band in shared memory; in runs of
// few slices C CTAs share it (deposit_part): its particles, added to a tile in
// global memory (DepTile) of which the last to finish writes the source, or the
// bands of a large tile.  The integer sums and the scale, hence the bits, are the
// same however a slice is shared.
constexpr int kDepThreads = 512;
constexpr double kDepUnit = 1073741824.0;  // 2^30
constexpr int kDepMaxWidth = 896;     // tile width bound: mixed ngrid <= 880
// Output cells per band (a multiple of 4) where two CTAs share an SM and where
// one has it: re and im planes, then the counts per base cell ((hb + 1) bw <=
// cells + width) in shared memory
constexpr int kDepCells2 = 9216, kDepCells1 = 18432;
constexpr size_t dep_smem(int cells) { return (size_t)(3 * cells + kDepMaxWidth) * 4; }
// Tile of one slice: `cells` sums im 2^32 + re, the counts per base cell
// (one row more), the bits of the largest charge weight, the CTAs done and, of a
// slice shared by bands, the largest number of contributions to a cell.
constexpr int kDepTileCells = 65536;  // at most
struct DepTile {
  unsigned long long* sum;
  int* hist;
  int* qmax;
  unsigned* done;
  int* mmax;
};
__host__ __device__ constexpr size_t dep_tile_bytes(int cells) {
  return (size_t)cells * 8 + (size_t)(cells + kDepMaxWidth) * 4 + 128;
}
__device__ __forceinline__ DepTile dep_tile(unsigned char* tiles, int cells, int bs) {
  DepTile t;
  t.sum = reinterpret_cast<unsigned long long*>(tiles + bs * dep_tile_bytes(cells));
  t.hist = reinterpret_cast<int*>(t.sum + cells);
  t.qmax = t.hist + cells + kDepMaxWidth;
  t.done = reinterpret_cast<unsigned*>(t.qmax + 1);
  t.mmax = t.qmax + 2;
  return t;
}

// Charge weight sqrt(faw2) / gamma of one particle (FP32).
__device__ __forceinline__ float dep_charge(const DepArgs& a, const float2 xy, const float dg) {
  const float dxu = xy.x - a.ax, dyu = xy.y - a.ay;
  // 1 + kx dx^2 + ky dy^2 + 2 (gradx dx + grady dy), every rounding explicit
  const float lin = __fmaf_rn(a.grady, dyu, __fmul_rn(a.gradx, dxu));
  const float faw2 = __fmaf_rn(__fmul_rn(a.kx, dxu), dxu,
                               __fmaf_rn(__fmul_rn(a.ky, dyu), dyu, __fmaf_rn(2.0f, lin, 1.0f)));
  return __fdividef(sqrtf(faw2), a.gref_f + dg);
}

// One field's source tile of one slice.
struct DepSlice {
  int bs, np, target;
  const float2* xy;
  const float* dg;
  const double* th;
  double scl;
  int bx0, by0, bw, bh;
  int m_use;     // bound M' of the contributions (0: no previous deposition)
  float q_use;   // bound q' of the charge weights (0: no previous deposition)
  MixField mf;
  float fh, inv_bw;
  __device__ __forceinline__ bool predicted() const {
    return m_use > 0 && q_use > 0.f && q_use < 3.0e38f;
  }
  // the predicted bounds' M' q': the scale is 2^30 / (M' q')
  __device__ __forceinline__ double bound() const { return (double)m_use * (double)q_use; }
};

// False (and no source, which thread 0 of the caller with `lead` writes): no
// particle in the grid, no current, or a tile the kernels do not take.
__device__ __forceinline__ bool dep_setup(const DepArgs& a, const DepField& F, const int bs,
                                          const bool lead, DepSlice& d) {
  d.bs = bs;
  const int64_t p0 = a.off[bs];
  d.np = (int)(a.off[bs + 1] - p0);  // at most kRunMaxNp per slice
  d.xy = a.xy + p0;
  d.dg = a.dg + p0;
  d.th = a.th + p0;
  d.target = (bs + F.first) % F.nslice;
  const int4 bb = F.bbox[bs];
  // M and qmax of this slice's previous deposition of this field bound the
  // contributions of the single-pass form
  const int mprev = F.mpred[bs];
  d.m_use = mprev > 0 ? mprev + (mprev >> 2) + 4 : 0;
  d.q_use = F.qpred[bs] * 1.015625f;
  d.scl = 0.0;
  if (d.np > 0) d.scl = F.kscl * a.current[bs] / (double)d.np;
  d.bx0 = bb.x;
  d.bw = bb.z - bb.x + 2;
  d.by0 = bb.y;
  d.bh = bb.w - bb.y + 2;
  const bool none = bb.z < 0 || d.scl == 0.0;
  if (!none && (d.bw & 1)) {  // even tile width keeps the rows 16-byte aligned
    ++d.bw;
    if (d.bx0 + d.bw > F.ld) --d.bx0;
  }
  const bool wide = !none && d.bw > kDepMaxWidth;  // excluded by g4b_run_create's ngrid limit
  if (lead && threadIdx.x == 0) {
    if (wide) atomicOr(a.err, kErrBadSlice);
    F.desc[d.target] = none || wide ? make_int4(0, 0, 0, 0) : make_int4(d.bx0, d.by0, d.bw, d.bh);
  }
  if (none || wide) return false;
  d.fh = (float)F.harm;
  d.inv_bw = 1.0f / (float)d.bw;
  d.mf.gridmax = F.gridmax;
  d.mf.dgrid = F.dgrid;
  d.mf.inv_dgrid = F.inv_dgrid;
  d.mf.n = F.n;
  return true;
}

// The rounded contributions of one particle of scaled charge weight q: (re, im)
// of the lower corners (ix, ix + 1), then of the upper ones.
__device__ __forceinline__ void dep_corners(const DepSlice& d, const float2 xy, const double th,
                                            const float q, int (&c)[8]) {
  float sn, cs;
  __sincosf(reduce_angle((double)d.fh * th), &sn, &cs);
  const float vre = sn * q, vim = cs * q;
  int ix, iy;
  float x0, y0;
  cell_f(d.mf, xy.x, xy.y, ix, iy, x0, y0);  // the weights
  const float w00 = x0 * y0, w10 = (1.f - x0) * y0, w01 = x0 * (1.f - y0),
              w11 = (1.f - x0) * (1.f - y0);
  c[0] = __float2int_rn(vre * w00);
  c[1] = __float2int_rn(vim * w00);
  c[2] = __float2int_rn(vre * w10);
  c[3] = __float2int_rn(vim * w10);
  c[4] = __float2int_rn(vre * w01);
  c[5] = __float2int_rn(vim * w01);
  c[6] = __float2int_rn(vre * w11);
  c[7] = __float2int_rn(vim * w11);
}

// Adds the particles [plow, phigh) of the slice to the rows ylo .. ylo + hb - 1:
// with `count` the counts per base cell (ext row iy - ylo + 1) and the largest
// charge weight (qloc), with `add` the contributions at scale Sf of charge
// weights capped at qc.  One particle per lane, the next one's loads in
// flight.  Four consecutive particles of one base cell (a quiet-start beamlet,
// nbins = 4 particles at one transverse position) are summed over their lanes,
// each of which adds one corner, with one count (the same integer sums).
// GLOBAL: to a DepTile; else to planes in shared memory.
template <int T, bool GLOBAL>
__device__ __forceinline__ void dep_pass(const DepArgs& a, const DepSlice& d, const int plow,
                                         const int phigh, const int ylo, const int hb, int* are,
                                         int* aim, unsigned long long* packed, int* hist,
                                         const bool count,
                                         const bool add, const float Sf, const float qc,
                                         float& qloc) {
  const int tid = threadIdx.x, l = tid & 31;
  const int bw = d.bw, nout = hb * bw;
  auto add2 = [&](int o, int re, int im) {
    if (GLOBAL) {
      atomicAdd(&packed[o], ((unsigned long long)(unsigned)im << 32) +
                                (unsigned long long)(long long)re);
    } else {
      atomicAdd(&are[o], re);
      atomicAdd(&aim[o], im);
    }
  };
  float2 nxy = make_float2(0.f, 0.f);
  float ndg = 0.f;
  double nth = 0.0;
  auto load = [&](int p) {
    if (p < phigh) {
      nxy = d.xy[p];
      ndg = d.dg[p];
      if (add) nth = d.th[p];
    }
  };
  load(plow + tid);
  for (int p = plow + tid; p - l < phigh; p += T) {  // whole warps
    const float2 xy = nxy;
    const float dg = ndg;
    const double th = nth;
    load(p + T);
    int cid = -1, ix, iy;
    float x0, y0;
    if (p < phigh && cell_f(d.mf, xy.x, xy.y, ix, iy, x0, y0) && iy + 1 >= ylo && iy < ylo + hb) {
      const int ex = ix - d.bx0;
      if (ex < 0 || ex > bw - 2) {
        if (count) atomicOr(a.err, kErrBadSlice);
      } else {
        cid = (iy - ylo + 1) * bw + ex;
      }
    }
    const int lead = __shfl_sync(0xffffffffu, cid, l & ~3);
    const unsigned match = __ballot_sync(0xffffffffu, cid >= 0 && cid == lead);
    const bool same = ((match >> (l & ~3)) & 15u) == 15u;
    if (count) {
      const int n = same ? ((l & 3) == 0 ? 4 : 0) : (cid >= 0 ? 1 : 0);
      if (n > 0) atomicAdd(&hist[cid], n);
    }
    // contributions to the lower corners (row ey - 1) and the upper ones, (re, im)
    int c[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (cid >= 0) {
      const float qraw = dep_charge(a, xy, dg);
      if (count) qloc = fmaxf(qloc, qraw);
      if (add) dep_corners(d, xy, th, fminf(qraw, qc) * Sf, c);
    }
    if (!add) continue;
    // a beamlet's sums: lane l ends with the corner of row (l & 2), column (l & 1)
    const bool up = (l & 2) != 0, right = (l & 1) != 0;
    int k[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      k[i] = (up ? c[4 + i] : c[i]) + __shfl_xor_sync(0xffffffffu, up ? c[i] : c[4 + i], 2);
    const int re = (right ? k[2] : k[0]) + __shfl_xor_sync(0xffffffffu, right ? k[0] : k[2], 1);
    const int im = (right ? k[3] : k[1]) + __shfl_xor_sync(0xffffffffu, right ? k[1] : k[3], 1);
    if (same) {
      if (up ? cid < nout : cid >= bw) add2((up ? cid : cid - bw) + (right ? 1 : 0), re, im);
    } else if (cid >= 0) {
      if (cid >= bw) {  // lower corners: output row ey = cid / bw - 1
        add2(cid - bw, c[0], c[1]);
        add2(cid - bw + 1, c[2], c[3]);
      }
      if (cid < nout) {  // upper corners: row ey + 1 inside the band
        add2(cid, c[4], c[5]);
        add2(cid + 1, c[6], c[7]);
      }
    }
  }
}

// Counts and contributions to shared memory by threads that take a group of four
// consecutive particles each (16-byte loads where the slice starts on a
// multiple of four): more work in flight per thread, for CTAs that have an SM,
// or half of one, to themselves at up to 128 registers.
template <int T>
__device__ __forceinline__ void dep_pass4(const DepArgs& a, const DepSlice& d, const int ylo,
                                          const int hb, int* are, int* aim, int* hist,
                                          const float Sf, const float qc, float& qloc) {
  const int bw = d.bw, nout = hb * bw;
  const bool wide = ((uintptr_t)d.dg & 15) == 0;  // d.dg + 4 g, hence d.xy and d.th too
  auto add8 = [&](int cid, const int* v) {
    if (cid >= bw) {  // lower corners: output row ey = cid / bw - 1
      const int o = cid - bw;
      atomicAdd(&are[o], v[0]);
      atomicAdd(&aim[o], v[1]);
      atomicAdd(&are[o + 1], v[2]);
      atomicAdd(&aim[o + 1], v[3]);
    }
    if (cid < nout) {  // upper corners: row ey + 1 inside the band
      atomicAdd(&are[cid], v[4]);
      atomicAdd(&aim[cid], v[5]);
      atomicAdd(&are[cid + 1], v[6]);
      atomicAdd(&aim[cid + 1], v[7]);
    }
  };
  for (int pg = 4 * threadIdx.x; pg < d.np; pg += 4 * T) {
    float2 lxy[4];
    float ldg[4];
    double lth[4];
    if (wide && pg + 3 < d.np) {
      const float4 u = *reinterpret_cast<const float4*>(d.xy + pg);
      const float4 v = *reinterpret_cast<const float4*>(d.xy + pg + 2);
      const float4 q = *reinterpret_cast<const float4*>(d.dg + pg);
      lxy[0] = make_float2(u.x, u.y);
      lxy[1] = make_float2(u.z, u.w);
      lxy[2] = make_float2(v.x, v.y);
      lxy[3] = make_float2(v.z, v.w);
      ldg[0] = q.x;
      ldg[1] = q.y;
      ldg[2] = q.z;
      ldg[3] = q.w;
      const double2 s = *reinterpret_cast<const double2*>(d.th + pg);
      const double2 t = *reinterpret_cast<const double2*>(d.th + pg + 2);
      lth[0] = s.x;
      lth[1] = s.y;
      lth[2] = t.x;
      lth[3] = t.y;
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (pg + u < d.np) {
          lxy[u] = d.xy[pg + u];
          ldg[u] = d.dg[pg + u];
          lth[u] = d.th[pg + u];
        }
      }
    }
    int cid[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      cid[u] = -1;
      int ix, iy;
      float wx, wy;
      if (pg + u < d.np && cell_f(d.mf, lxy[u].x, lxy[u].y, ix, iy, wx, wy) && iy + 1 >= ylo &&
          iy < ylo + hb) {
        const int ex = ix - d.bx0;
        if (ex < 0 || ex > bw - 2) {
          atomicOr(a.err, kErrBadSlice);
        } else {
          cid[u] = (iy - ylo + 1) * bw + ex;
        }
      }
    }
    const bool same = cid[0] >= 0 && cid[1] == cid[0] && cid[2] == cid[0] && cid[3] == cid[0];
    if (same) {
      atomicAdd(&hist[cid[0]], 4);
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (cid[u] >= 0) atomicAdd(&hist[cid[u]], 1);
    }
    int sum[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (cid[u] < 0) continue;
      const float qraw = dep_charge(a, lxy[u], ldg[u]);
      qloc = fmaxf(qloc, qraw);
      int c[8];
      dep_corners(d, lxy[u], lth[u], fminf(qraw, qc) * Sf, c);
      if (same) {
#pragma unroll
        for (int k = 0; k < 8; ++k) sum[k] += c[k];
      } else {
        add8(cid[u], c);
      }
    }
    if (same) add8(cid[0], sum);
  }
}

// Block maximum of M and of the charge weight.
template <int T>
__device__ __forceinline__ void dep_max(int& M, float& q) {
  __shared__ int wsum[T / 32];
  __shared__ float wmax[T / 32];
  M = __reduce_max_sync(0xffffffffu, M);
  for (int o = 16; o > 0; o >>= 1) q = fmaxf(q, __shfl_xor_sync(0xffffffffu, q, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    wsum[threadIdx.x >> 5] = M;
    wmax[threadIdx.x >> 5] = q;
  }
  __syncthreads();
  M = wsum[0];
  q = wmax[0];
  for (int i = 1; i < T / 32; ++i) {
    M = max(M, wsum[i]);
    q = fmaxf(q, wmax[i]);
  }
}

// Two neighbouring source cells (bw and the cell counts are even, the rows
// 16-byte aligned).
__device__ __forceinline__ void dep_write(float2* out, int2 re, int2 im, double unscale) {
  *reinterpret_cast<float4*>(out) =
      make_float4((float)((double)re.x * unscale), (float)((double)im.x * unscale),
                  (float)((double)re.y * unscale), (float)((double)im.y * unscale));
}

// The rare passes (counts alone, or the contributions alone), out of line.
template <int T>
__device__ __noinline__ float dep_rare(const DepArgs& a, const DepSlice d, const int ylo,
                                       const int hb, int* are, int* aim, int* hist,
                                       const bool count, const float Sf, const float qc) {
  float q = 0.f;
  dep_pass<T, false>(a, d, 0, d.np, ylo, hb, are, aim, nullptr, hist, count, !count, Sf, qc, q);
  return q;
}

// True in the CTA that comes last of the C that share a slice: what the others
// wrote before is then visible to it, and each has read the prediction.
__device__ __forceinline__ bool dep_last(const DepTile& t, const int C) {
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(t.done, 1u) == (unsigned)C - 1u;
  __syncthreads();
  if (last) __threadfence();
  return last != 0;
}

// One field of a slice by a whole CTA, band by band of at most CELLS cells in
// shared memory; FOUR: by dep_pass4.  With a prediction one pass takes counts,
// qmax and contributions at the scale of the predicted bounds; it is kept if
// neither counted bound exceeds its prediction (then no cell sum can have
// overflowed and no charge was capped), else the contributions are redone at
// the exact scale 2^30 / (M qmax).  Without one, a first pass only counts.  M
// and qmax are the slice's, whatever its bands.  With C > 1 (and a prediction)
// CTA `rank` of C takes the bands rank, rank + C, ..., and the last of them to
// finish goes on with the slice's M and qmax, alone.
template <int T, bool FOUR, int CELLS>
__device__ __forceinline__ void deposit_field(const DepArgs& a, const DepField& F,
                                              const DepSlice& d, unsigned char* smem, int rank = 0,
                                              int C = 1) {
  const int tid = threadIdx.x, bw = d.bw;
  int* are = reinterpret_cast<int*>(smem);        // [hb * bw] real parts
  int* aim = are + CELLS;                         // [hb * bw] imaginary parts
  int* hist = aim + CELLS;                        // [(hb + 1) * bw] counts per base cell
  const int hband = max(1, CELLS / bw);           // bw <= ngrid + 1 < CELLS
  auto zero = [&](int* p, int n) {
    for (int i = tid; i < (n + 3) >> 2; i += T) reinterpret_cast<int4*>(p)[i] = make_int4(0, 0, 0, 0);
  };
  int M = 0;
  float qm = 0.f;
  bool count = true, add = d.predicted();
  double B = d.bound();  // the scale is kDepUnit / B
  float qc = d.q_use;
  for (;;) {
    const float Sf = (float)(kDepUnit / B);
    const double unscale = d.scl * (B * (1.0 / kDepUnit));
    for (int yb = rank * hband; yb < d.bh; yb += C * hband) {
      const int hb = min(hband, d.bh - yb), nout = hb * bw;
      __syncthreads();
      if (count) zero(hist, (hb + 1) * bw);
      if (add) {
        zero(are, nout);
        zero(aim, nout);
      }
      __syncthreads();
      if (!(count && add))
        qm = fmaxf(qm, dep_rare<T>(a, d, d.by0 + yb, hb, are, aim, hist, count, Sf, qc));
      else if (FOUR)
        dep_pass4<T>(a, d, d.by0 + yb, hb, are, aim, hist, Sf, qc, qm);
      else
        dep_pass<T, false>(a, d, 0, d.np, d.by0 + yb, hb, are, aim, nullptr, hist, true, true, Sf,
                           qc, qm);
      __syncthreads();
      // the cells' sums, and the largest number M of contributions any output
      // cell receives (its four base cells' counts); row of cell o: (o + 1/2)
      // / bw in FP32 is never within nout 2^-23 / bw of an integer boundary,
      // so the truncation is exact
      float2* out = F.src + (size_t)d.target * F.cap + (size_t)yb * bw;
      for (int o = 2 * tid; o < nout; o += 2 * T) {
        if (add)
          dep_write(out + o, *reinterpret_cast<const int2*>(are + o),
                    *reinterpret_cast<const int2*>(aim + o), unscale);
        if (!count) continue;
        const int x = o - (int)(((float)o + 0.5f) * d.inv_bw) * bw;
        const int2 up = *reinterpret_cast<const int2*>(hist + o),
                   dn = *reinterpret_cast<const int2*>(hist + o + bw);
        const int left = x > 0 ? hist[o - 1] + hist[o + bw - 1] : 0;
        M = max(M, max(left + up.x + dn.x, up.x + dn.x + up.y + dn.y));
      }
    }
    if (!count) break;
    dep_max<T>(M, qm);
    if (C > 1) {
      const DepTile t = dep_tile(F.tiles, F.tile_cells, d.bs);
      if (tid == 0) {
        atomicMax(t.mmax, M);
        atomicMax(t.qmax, __float_as_int(qm));
      }
      if (!dep_last(t, C)) return;
      M = __ldcg(t.mmax);
      qm = __int_as_float(__ldcg(t.qmax));
      __syncthreads();
      if (tid == 0) {
        *t.mmax = 0;
        *t.qmax = 0;
        *t.done = 0;
      }
      rank = 0;
      C = 1;
    }
    if (M == 0 || !(qm > 0.f) || !(qm < 3.0e38f)) {
      if (M > 0) atomicOr(a.err, kErrFixedRange);  // non-finite charge
      float2* out = F.src + (size_t)d.target * F.cap;
      for (int i = tid; i < d.bh * bw; i += T) out[i] = make_float2(0.f, 0.f);
      qm = 0.f;
      break;
    }
    if (add && M <= d.m_use && qm <= d.q_use) break;
    count = false;
    add = true;
    B = (double)M * (double)qm;
    qc = qm;
  }
  if (tid == 0) {
    F.mpred[d.bs] = M;
    if (qm > 0.f) F.qpred[d.bs] = qm;
  }
}

template <int T, bool FOUR, int CELLS>
__device__ __forceinline__ void deposit_slice(const DepArgs& a, const int bs, unsigned char* smem) {
  for (int fi = 0; fi < a.nfield; ++fi) {
    const DepField& F = a.f[fi];
    DepSlice d;
    if (F.do_source && dep_setup(a, F, bs, true, d)) deposit_field<T, FOUR, CELLS>(a, F, d, smem);
  }
}

// Part `rank` of C of a slice in runs of few slices, by one of three ways:
//   tile: each CTA adds its 1/C of the particles to the slice's DepTile; the one
//   whose count comes last reads it, writes the source and leaves the tile zero
//   for the next launch;
//   bands: the bands of a tile of several are shared out (deposit_field);
//   alone: CTA 0 does a tile of one band in shared memory.
// A shared field without a prediction, one whose prediction fails and one without
// a finite charge are done by the CTA that comes last, alone.
// Where the lines lie (us per graph step; [ ]: two CTAs per slice, bands dealt in
// turn).  Adds to L2 cost a particle more than adds to shared memory, four times
// over where its beamlet is not four neighbours of one slice, and the tile costs
// its reading; the bands cost a pass over all particles each.
//   One band, tile / alone: 1 x 2048 (129^2) 20.1 / 19.3 [21.6], 1 x 3000 (151^2)
//   20.1 / 21.9, 12 x 8192 (201^2) 28.2 / 31.8 [33.4], 12 x 32768 66.2 / 69.0 [70];
//   from 13 slices by the grouping (dep_grouped): beamlets of four, 16 x 32768 46
//   / 64 [71], 21 x 8192 32.1 / 32.9 [36.2]; others, 16 x 16384 (151^2) 48 / 41
//   [42], 21 x 32768 105 / 69 [74].
//   Several bands, tile / bands: 1 x 6000 (255^2) 57 / 31 [67], 21 x 6000 76 / 41
//   [78], 1 x 60000 58 / 80 [223], 8 x 60000 105 / 105 [273]; more than 65536
//   cells, alone / bands: 1 x 6000 (401^2) 123 / 33 [113], 21 x 159 / 72 [154].
constexpr int kDepShareNp = 2560, kDepShareC = 11;
constexpr int kDepShareNp2 = 32768, kDepShareC2 = 16;

// Do the first 32 groups of four particles of a slice mostly share a cell (the
// beamlets of a quiet start)?  The same answer in every warp.
__device__ __forceinline__ bool dep_grouped(const DepSlice& d) {
  const int p = 4 * (threadIdx.x & 31);  // d.np is larger
  int cell[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const float2 xy = d.xy[p + u];
    int ix, iy;
    float wx, wy;
    cell[u] = cell_f(d.mf, xy.x, xy.y, ix, iy, wx, wy) ? iy * d.mf.n + ix : -1;
  }
  const bool same = cell[0] == cell[1] && cell[0] == cell[2] && cell[0] == cell[3];
  return __popc(__ballot_sync(0xffffffffu, same)) >= 24;
}

template <int T>
__device__ __forceinline__ void deposit_part(const DepArgs& a, const int bs, const int rank,
                                             const int C, unsigned char* smem) {
  const int tid = threadIdx.x;
  for (int fi = 0; fi < a.nfield; ++fi) {
    const DepField& F = a.f[fi];
    DepSlice d;
    if (!F.do_source || !dep_setup(a, F, bs, rank == 0, d)) continue;
    const int bw = d.bw, nout = d.bh * bw, nbase = (d.bh + 1) * bw;
    const DepTile t = dep_tile(F.tiles, F.tile_cells, bs);
    const bool bands = nout > kDepCells1;
    const bool tile = bands ? C >= kDepShareC2 && d.np >= kDepShareNp2 && nout <= F.tile_cells
                            : d.np >= kDepShareNp && (C >= kDepShareC || dep_grouped(d));
    int r = 0, c = 1;  // deposit_field's share, unless the tile does
    if (!bands && !tile) {
      if (rank > 0) continue;  // CTA 0's
    } else if (!d.predicted()) {
      if (!dep_last(t, C)) continue;
      if (tid == 0) *t.done = 0;
    } else if (!tile) {
      r = rank;
      c = C;
    } else {
      const int share = (((d.np + 3) >> 2) + C - 1) / C * 4, plow = rank * share;
      float qm = 0.f;
      dep_pass<T, true>(a, d, plow, min(d.np, plow + share), d.by0, d.bh, nullptr, nullptr, t.sum,
                        t.hist, true, true, (float)(kDepUnit / d.bound()), d.q_use, qm);
      for (int o = 16; o > 0; o >>= 1) qm = fmaxf(qm, __shfl_xor_sync(0xffffffffu, qm, o));
      if ((tid & 31) == 0 && qm > 0.f) atomicMax(t.qmax, __float_as_int(qm));
      if (!dep_last(t, C)) continue;
      float2* out = F.src + (size_t)d.target * F.cap;
      const double unscale = d.scl * (d.bound() * (1.0 / kDepUnit));
      int M = 0;
      for (int o = 2 * tid; o < nout; o += 2 * T) {
        const longlong2 v = __ldcg(reinterpret_cast<const longlong2*>(t.sum + o));
        const int x = o - (int)(((float)o + 0.5f) * d.inv_bw) * bw;
        const int2 up = __ldcg(reinterpret_cast<const int2*>(t.hist + o)),
                   dn = __ldcg(reinterpret_cast<const int2*>(t.hist + o + bw));
        const int left = x > 0 ? __ldcg(t.hist + o - 1) + __ldcg(t.hist + o + bw - 1) : 0;
        const int2 re = make_int2((int)(unsigned)v.x, (int)(unsigned)v.y);
        dep_write(out + o, re,
                  make_int2((int)((v.x - re.x) >> 32), (int)((v.y - re.y) >> 32)), unscale);
        M = max(M, max(left + up.x + dn.x, up.x + dn.x + up.y + dn.y));
      }
      qm = __int_as_float(__ldcg(t.qmax));
      dep_max<T>(M, qm);  // (every cell has been read)
      for (int o = 2 * tid; o < nbase; o += 2 * T) {
        if (o < nout) *reinterpret_cast<int4*>(t.sum + o) = make_int4(0, 0, 0, 0);
        *reinterpret_cast<int2*>(t.hist + o) = make_int2(0, 0);
      }
      if (tid == 0) {
        *t.qmax = 0;
        *t.done = 0;
      }
      // without a finite positive charge too deposit_field goes on: it reports that
      if (M <= d.m_use && qm > 0.f && qm <= d.q_use) {
        if (tid == 0) {
          F.mpred[bs] = M;
          F.qpred[bs] = qm;
        }
        continue;
      }
    }
    deposit_field<T, true, kDepCells1>(a, F, d, smem, r, c);
  }
}

// A CTA per slice.  BESIDE: lets the next kernel (beam_diag_kernel) start
// beside this one, once every CTA runs or has ended.
template <bool BESIDE>
__global__ void __launch_bounds__(kDepThreads, 2)
    deposit_kernel(const __grid_constant__ DepArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  ptx::pdl_wait();
  if (BESIDE) ptx::pdl_launch_dependents();
  deposit_slice<kDepThreads, false, kDepCells2>(a, blockIdx.x, smem);
}

// Fewer slices than SMs: per slice one CTA for the beam diagnostics and the
// others for the deposition, side by side.
struct DepDiagLaunch {
  DepArgs d;
  BeamDiagArgs b;
  int parts;
};

template <int NB, int T, bool SHARED>
__device__ __forceinline__ void deposit_diag_part(const DepArgs& d, const BeamDiagArgs& b,
                                                  const int bs, const int part, const int parts,
                                                  unsigned char* smem) {
  if (part == parts - 1) {
    DiagGroups<NB>& G = *reinterpret_cast<DiagGroups<NB>*>(smem);
    diag_groups<NB>(b, bs, threadIdx.x >> 5, T / 32, G);
    __syncthreads();
    diag_record<NB, T>(b, bs, G);
  } else if (SHARED) {
    deposit_part<T>(d, bs, part, parts - 1, smem);
  } else {
    deposit_slice<T, true, T == 512 ? kDepCells1 : kDepCells2>(d, bs, smem);
  }
}

template <int NB, int T, bool SHARED>
__global__ void __launch_bounds__(T, 512 / T)
    deposit_diag_kernel(const __grid_constant__ DepDiagLaunch a) {
  extern __shared__ __align__(128) unsigned char smem[];
  ptx::pdl_wait();
  deposit_diag_part<NB, T, SHARED>(a.d, a.b, blockIdx.x / a.parts, blockIdx.x % a.parts, a.parts,
                                   smem);
}

// Batched forms: items[i] = (run, slice of that run).
struct DepBatchArgs {
  const DepArgs* args;
  const int2* items;
  const int* nitems;
};

__global__ void __launch_bounds__(kDepThreads, 2)
    deposit_batch_kernel(const __grid_constant__ DepBatchArgs b) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int nitems = *b.nitems;
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const int2 w = b.items[it];
    deposit_slice<kDepThreads, false, kDepCells2>(b.args[w.x], w.y, smem);
    __syncthreads();
  }
}

struct DiagBatchArgs {
  const BeamDiagArgs* args;
  const int2* items;
  const int* nitems;
};

template <int NB, bool SHARED>
__global__ void __launch_bounds__(512, 1)
    deposit_diag_batch_kernel(const __grid_constant__ DepBatchArgs b, const BeamDiagArgs* diag,
                              const int parts) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int2 w = b.items[blockIdx.x / parts];
  deposit_diag_part<NB, 512, SHARED>(b.args[w.x], diag[w.x], w.y, blockIdx.x % parts, parts, smem);
}

template <int NB>
__global__ void __launch_bounds__(kDiagThreads, 2)
    beam_diag_batch_kernel(const __grid_constant__ DiagBatchArgs b) {
  __shared__ DiagGroups<NB> G;
  const int nitems = *b.nitems;
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const int2 w = b.items[it];
    const BeamDiagArgs& a = b.args[w.x];
    diag_groups<NB>(a, w.y, threadIdx.x >> 5, kDiagThreads / 32, G);
    __syncthreads();
    diag_record<NB, kDiagThreads>(a, w.y, G);
    __syncthreads();
  }
}

// How a launch over `nslice` slices is split.  parts > 0: that many CTAs per
// slice, one of them for the diagnostics, of T threads: one CTA of 512 per SM
// or two of 256; parts > 2: the deposition shared out (deposit_part).  Else
// one CTA per slice for the deposition and the diagnostics in a kernel of their
// own: beside it, or in a branch of the graph where the slices fill the GPU
// twice.  A deposition waits on its loads, conversions and shared-memory atomics
// in turn, so what pays is warps per SM: 32 with a particle per lane (64
// registers) where two CTAs share an SM; four particles per thread at 128
// registers where there is one.  A pair of 256 threads has half the band and half
// the threads for a tile of several bands, and saves time only on small slices.
// Measured, us per graph step, two CTAs per slice with bands dealt in turn /
// pairs of 256 / of 512 / one CTA per slice:
//   22 x 8192 (201^2) 37.9 / - / 33.4 / -, 74 x 8192 63 / 73 / 52 / 80;
//   75 x 2048 (129^2) 31 / 29 / 31 / 30, 147 x 500 (65^2) 24 / 22 / 26 / 26;
//   75 x 8192 69 / 62 / 60 / 61, 75 x 6000 (255^2, four bands) 141 / 173 / 110 /
//   142, 90 x 32768 165 / 182 / 137 / 167, 75 x 3000 (151^2) 43 / 40 / 41 / 41;
//   110 x 8192 87 / 79 / 77 / 75, 123 x 3000 56 / 53 / 57 / 52, 147 x 6000 (255^2)
//   199 / 236 / 188 / 184, 147 x 32768 219 / 223 / 200 / 199;
//   200 x 8192 139 / 136 / 139 / 128; 1024: the deposition 97 us (121).
constexpr int kSplitMaxParts = 17;
struct DepSplit {
  int parts, T;
  size_t smem() const { return dep_smem(T == 512 ? kDepCells1 : kDepCells2); }
};
// Shared out: up to 21 slices.
static DepSplit dep_split_few(int nslice, int sm_count) {
  const int parts = std::min(kSplitMaxParts, sm_count / nslice);
  return parts >= 7 ? DepSplit{parts, 512} : DepSplit{0, 0};
}
// max_np: particles of the largest slice.
static DepSplit dep_split(int nslice, int max_np, int sm_count) {
  const DepSplit few = dep_split_few(nslice, sm_count);
  if (few.parts > 0) return few;
  if (2 * nslice <= sm_count) return {2, 512};
  if (nslice < sm_count && max_np <= 2048) return {2, 256};
  if (3 * nslice < 2 * sm_count) return {2, 512};
  return {0, 0};
}

// The same for the slices of a batch, whose particle counts differ: a large slice
// in a narrow CTA is the whole launch's length, so pairs of 512 threads up to four
// slices per SM, the hardware dealing them out as SMs come free; beyond, the
// persistent kernels (32 warps per SM) win on slices of one size.  Measured, us
// per step (pairs of 256 threads to 147 slices and persistent kernels above):
//   steady-state runs of 2048-32768 particles: 100 of them 222 (322), 140 259
//   (343), 148 279 (412), 256 436 (515), 500 753 (838);
//   runs of 100 slices of 8192: two 209 (253), four 370 (425); four runs of 200
//   slices of 4096 463 (448).
static DepSplit dep_split_batch(int nslice, int sm_count) {
  const DepSplit few = dep_split_few(nslice, sm_count);
  if (few.parts > 0) return few;
  return nslice <= 4 * sm_count ? DepSplit{2, 512} : DepSplit{0, 0};
}

// The kernels of a split: one bunching harmonic or any number.
using DepDiagKernel = void (*)(DepDiagLaunch);
static DepDiagKernel dep_diag_kernel(bool one, DepSplit s) {
  if (s.parts > 2) return one ? deposit_diag_kernel<1, 512, true> : deposit_diag_kernel<kMaxBunch, 512, true>;
  if (s.T == 512) return one ? deposit_diag_kernel<1, 512, false> : deposit_diag_kernel<kMaxBunch, 512, false>;
  return one ? deposit_diag_kernel<1, 256, false> : deposit_diag_kernel<kMaxBunch, 256, false>;
}
using DepDiagBatchKernel = void (*)(DepBatchArgs, const BeamDiagArgs*, int);
static DepDiagBatchKernel dep_diag_batch_kernel(bool one, DepSplit s) {
  if (s.parts > 2) return one ? deposit_diag_batch_kernel<1, true> : deposit_diag_batch_kernel<kMaxBunch, true>;
  return one ? deposit_diag_batch_kernel<1, false> : deposit_diag_batch_kernel<kMaxBunch, false>;
}

// ---------------------------------------------------------- diag finalize --
// Field diagnostics per beam slice is = (nslice + storage - first) % nslice
// (src/Core/DiagnosticCUDA.cpp:320) from the pass-Y band partials.
struct FinalizeArgs {
  const double* part[kRunFields];  // [nslice][nband][9]
  int4* bbox[kRunFields];
  int nband[kRunFields];
  int first_after[kRunFields];
  int nfield, nslice;
  double* field_hist;       // [nfield][nslice][9] for this step
};

// Per-slice reductions in fixed order: field diagnostics per beam slice
// is = (nslice + storage - first) % nslice (src/Core/DiagnosticCUDA.cpp:320)
// from the pass-Y band partials (one thread per slice and quantity, adding
// the bands in order); also resets the deposition boxes for the next step.
__device__ __forceinline__ void finalize_range(const FinalizeArgs& a, int i0, int stride) {
  const int nf = a.nfield * a.nslice;
  for (int i = i0; i < 9 * nf + nf; i += stride) {
    if (i < 9 * nf) {
      const int j = i / 9, q = i - 9 * j;
      const int f = j / a.nslice, s = j - f * a.nslice;
      const double* p = a.part[f] + (size_t)s * a.nband[f] * 9 + q;
      const int nbf = a.nband[f];
      double v = 0.0, vc = 0.0;  // compensated sum of the bands, in band order
      for (int b0 = 0; b0 < nbf; b0 += 32) {  // up to 32 loads in flight
        const int m = min(32, nbf - b0);
        double t[32];
#pragma unroll
        for (int k = 0; k < 32; ++k) t[k] = k < m ? p[(b0 + k) * 9] : 0.0;
#pragma unroll
        for (int k = 0; k < 32; ++k)
          if (k < m) ptx::csum_add(v, vc, t[k]);
      }
      v += vc;
      const int is = (a.nslice + s - a.first_after[f]) % a.nslice;
      a.field_hist[((size_t)f * a.nslice + is) * 9 + q] = v;
    } else {
      const int j = i - 9 * nf;
      const int f = j / a.nslice, s = j - f * a.nslice;
      a.bbox[f][s] = make_int4(1 << 30, 1 << 30, -1, -1);
    }
  }
}

__global__ void diag_finalize_kernel(const __grid_constant__ FinalizeArgs a) {
  ptx::pdl_wait();
  finalize_range(a, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// Batched form: one CTA per run at a time.
__global__ void finalize_batch_kernel(const FinalizeArgs* args, const int* nruns) {
  const int n = *nruns;
  for (int r = blockIdx.x; r < n; r += gridDim.x) finalize_range(args[r], threadIdx.x, blockDim.x);
}

// Particle conversions between FP64 host arrays (x, y, px, py, gamma, each
// `stride` apart in the staging buffer) and the mixed form's state.
__global__ void beam_f64_to_mixed(const double* stage, size_t stride, size_t m, float gf,
                                  float2* xy, float2* pxy, float* dg) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < m;
       i += (size_t)gridDim.x * blockDim.x) {
    xy[i] = make_float2((float)stage[i], (float)stage[stride + i]);
    pxy[i] = make_float2((float)stage[2 * stride + i], (float)stage[3 * stride + i]);
    dg[i] = (float)(stage[4 * stride + i] - (double)gf);
  }
}

__global__ void beam_mixed_to_f64(const float2* xy, const float2* pxy, const float* dg,
                                  double gf, size_t m, double* stage, size_t stride) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < m;
       i += (size_t)gridDim.x * blockDim.x) {
    const float2 a = xy[i], b = pxy[i];
    stage[i] = a.x;
    stage[stride + i] = a.y;
    stage[2 * stride + i] = b.x;
    stage[3 * stride + i] = b.y;
    stage[4 * stride + i] = gf + (double)dg[i];
  }
}

static PlaneMapF plane_map_f(double strength, double offset) {
  PlaneMapF m{0, (float)strength, 0.f};
  if (strength == 0.0) return m;
  m.offset = (float)(offset / strength);
  m.mode = strength > 0.0 ? 1 : 2;
  return m;
}

}  // namespace g4b

using namespace g4b;

struct StepPlan {
  g4b_step st;
  double fc[kRunFields];
  int first_before[kRunFields], first_after[kRunFields];
  int zero_start[kRunFields], zero_count[kRunFields];
  int adi_index[kRunFields];
};

struct RunFieldState {
  g4b_field* f = nullptr;
  std::vector<g4b_adi*> adis;   // one factorisation per distinct delz
  std::vector<double> adi_delz;
  int harm = 1;
  int4* d_bbox = nullptr;
  int* d_mpred = nullptr;       // [nslice] deposition contribution bound per slice
  float* d_qpred = nullptr;     // [nslice] largest charge weight of the last deposition
  unsigned char* d_tiles = nullptr;  // [nslice] DepTile of tile_cells (runs of few slices)
  int tile_cells = 0;
  double* d_part = nullptr;
  int nband = 0;
  double accuslip = 0.0;        // host slippage model
  int first = 0;
};

struct g4b_run {
  g4b_ctx* ctx = nullptr;
  g4b_run_desc desc{};
  int nslice = 0, nfield = 0;
  int64_t npart = 0, max_np = 0;
  int64_t* d_off = nullptr;
  int4* d_chunks = nullptr;
  int nchunk = 0;
  float2 *xy = nullptr, *pxy = nullptr;
  float* dg = nullptr;
  double* th = nullptr;
  double *d_current = nullptr, *d_eloss = nullptr;
  std::vector<double> h_current;
  RunFieldState fs[kRunFields];
  // lattice
  std::vector<g4b_step> steps;
  std::vector<double> fc;   // [nstep][nfield]
  std::vector<double> slip;
  // history of diagnostics: per step beam [nslice][rec] then fields
  double* d_hist = nullptr;
  // second stream and fork / join events of a captured step (diagnostics branch)
  cudaStream_t aux = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  bool capturing = false;
  int hist_steps = 0;
  size_t rec_beam = 0, step_doubles = 0;
  // cached graph
  cudaGraphExec_t gexec = nullptr;
  int g_first = -1, g_n = 0;
  std::vector<int> g_state;
  uint64_t bytes = 0;
};

// Chicane transfer matrix shared with the drop-in tracking (row-major 4x4).
void g4b_chicane_matrix(double angle, double lb, double ld, double lt, double* m);

namespace {

constexpr int kRunChunk = 2 * kStepThreads;  // particles per beam-step CTA

// Every argument of one lattice step of one run.
struct StepArgs {
  bool has_beam;
  BeamStepArgs bs;
  DepArgs dd;
  BeamDiagArgs bd;
  AdiPlan adi[kRunFields];
  FinalizeArgs fa;
};

int plan_step(g4b_run* r, int i, StepPlan& p) {
  p.st = r->steps[i];
  for (int f = 0; f < r->nfield; ++f) {
    RunFieldState& F = r->fs[f];
    p.fc[f] = r->fc[(size_t)i * r->nfield + f];
    p.first_before[f] = F.first;
    // slippage model of ControlCUDA::applySlippage (src/Core/ControlCUDA.cpp:148-252)
    int zs = 0, zc = 0;
    if (r->desc.time_run) {
      F.accuslip += r->slip[i];
      const int ns = r->nslice;
      int direction = 1;
      while (std::fabs(F.accuslip) > r->desc.sample * 0.8) {
        direction = F.accuslip < 0 ? -1 : 1;
        F.accuslip -= r->desc.sample * direction;
        int last = (F.first + ns - 1) % ns;
        if (direction < 0) last = (last + 1) % ns;
        if (!r->desc.periodic) {
          if (zc == 0) {
            zs = last;
            zc = 1;
          } else if (direction > 0 && (last + 1) % ns == zs) {
            zs = last;
            ++zc;
          } else if (direction < 0 && (zs + zc) % ns == last) {
            ++zc;
          } else {
            return fail(G4B_ERR_RANGE, "g4b_run: slippage changes direction within one step");
          }
        }
        F.first = last;
        if (direction < 0) F.first = (last + 1) % ns;
      }
    }
    p.zero_start[f] = zs;
    p.zero_count[f] = std::min(zc, r->nslice);
    p.first_after[f] = F.first;
    int k = -1;
    for (size_t j = 0; j < F.adi_delz.size(); ++j)
      if (F.adi_delz[j] == p.st.delz) k = (int)j;
    if (k < 0) return fail(G4B_ERR_STATE, "g4b_run: step length without a factorisation");
    p.adi_index[f] = k;
  }
  return G4B_OK;
}

// Resolves every kernel argument of lattice step i (plan p) without
// launching anything; the single-run path and the batch engine launch them.
int build_step(g4b_run* r, int i, const StepPlan& p, StepArgs& L) {
  g4b_ctx* c = r->ctx;
  L = StepArgs{};
  const g4b_step& st = p.st;
  const double gref = r->desc.gamma_ref;
  // particles store dg = gamma - (float)gamma_ref; every kernel rebuilds gamma
  // from that same FP32-rounded reference
  const double gbase = (double)(float)gref;
  // K1
  if (r->npart > 0) {
    BeamStepArgs a{};
    a.xy = r->xy;
    a.pxy = r->pxy;
    a.dg = r->dg;
    a.th = r->th;
    a.chunks = r->d_chunks;
    a.eloss = r->d_eloss;
    a.nfield = r->nfield;
    double xks_local = 1.0;
    for (int f = 0; f < r->nfield; ++f) {
      const RunFieldState& F = r->fs[f];
      MixField& m = a.f[f];
      m.cells = static_cast<const float2*>(F.f->a);
      m.first = p.first_before[f];
      m.n = F.f->ngrid;
      m.ld = F.f->ld;
      m.nslice = r->nslice;
      m.harm = F.harm;
      m.do_source = st.in_undulator && (F.harm % 2) == 1;
      m.gridmax = (float)F.f->gridmax;
      m.dgrid = (float)F.f->dgrid;
      m.inv_dgrid = (float)(1.0 / F.f->dgrid);
      m.rtmp = (float)(p.fc[f] / F.f->xks);
      m.bbox = F.d_bbox;
      xks_local = F.f->xks / (double)F.harm;
    }
    a.gref = gbase;
    a.gref_f = (float)gref;
    a.xks = xks_local;
    a.zt0 = (float)(-2.0 / xks_local);
    a.xku = st.ku != 0.0 ? st.ku : xks_local * 0.5 / gref / gref;
    a.delz = st.delz;
    a.half = (float)(0.5 * st.delz);
    a.autophase = st.autophase;
    a.aw = (float)st.aw;
    a.aw2 = (float)(st.aw * st.aw);
    a.ax = (float)st.ax;
    a.ay = (float)st.ay;
    a.kx = (float)st.kx;
    a.ky = (float)st.ky;
    a.gradx = (float)st.gradx;
    a.grady = (float)st.grady;
    const double betpar0 = std::sqrt(1 - (1 + st.aw * st.aw) / gref / gref);
    const double quad = st.qf * gref;
    const double qnatx = st.kx * st.aw * st.aw / gref / betpar0;
    const double qnaty = st.ky * st.aw * st.aw / gref / betpar0;
    a.xm = plane_map_f(quad + qnatx, quad * st.dqx + qnatx * st.ax);
    a.ym = plane_map_f(-quad + qnaty, -quad * st.dqy + qnaty * st.ay);
    if (st.chic_angle != 0) {
      // chicane matrix from the drop-in path's builder (TrackBeamCUDA.cpp:93-148)
      double m[16];
      g4b_chicane_matrix(st.chic_angle, st.chic_lb, st.chic_ld, st.chic_lt, m);
      a.pre = 1;
      a.m00 = (float)m[0];
      a.m01 = (float)m[1];
      a.m10 = (float)m[4];
      a.m11 = (float)m[5];
      a.m22 = (float)m[10];
      a.m23 = (float)m[11];
      a.m32 = (float)m[14];
      a.m33 = (float)m[15];
      const double ang = st.chic_angle, lb = st.chic_lb, ld = st.chic_ld;
      double r56 = (4 * lb / std::sin(ang) * (1 - ang / std::tan(ang)) +
                    2 * ld * std::tan(ang) / std::cos(ang)) * ang;
      a.r56 = r56 * 4 * std::asin(1.0) / r->desc.lambda0 / gref;
      a.r56_off = gbase - gref;  // gamma - gamma0 = dg + (gbase - gamma0)
      a.has_r56 = 1;
    }
    if (st.cx != 0 || st.cy != 0) {
      a.post = 1;
      a.cx = (float)(st.cx * gref);
      a.cy = (float)(st.cy * gref);
    }
    a.err = c->d_error;
    L.has_beam = true;
    L.bs = a;
  }
  // K2
  double* step_hist = r->d_hist + (size_t)(i % r->hist_steps) * r->step_doubles;
  {
    BeamDiagArgs b{};
    b.xy = r->xy;
    b.pxy = r->pxy;
    b.dg = r->dg;
    b.th = r->th;
    b.off = r->d_off;
    b.nbunch = r->desc.nbunch;
    b.need_aux = 1;
    b.gref = gbase;
    b.beam_hist = step_hist;
    L.bd = b;
    DepArgs a{};
    a.xy = r->xy;
    a.dg = r->dg;
    a.th = r->th;
    a.off = r->d_off;
    a.current = r->d_current;
    a.nfield = r->nfield;
    a.ax = (float)st.ax;
    a.ay = (float)st.ay;
    a.kx = (float)st.kx;
    a.ky = (float)st.ky;
    a.gradx = (float)st.gradx;
    a.grady = (float)st.grady;
    a.delz = st.delz;
    a.gref_f = (float)gbase;
    a.err = c->d_error;
    for (int f = 0; f < r->nfield; ++f) {
      const RunFieldState& F = r->fs[f];
      DepField& d = a.f[f];
      d.src = static_cast<float2*>(F.f->src);
      d.desc = F.f->desc;
      d.bbox = F.d_bbox;
      d.mpred = F.d_mpred;
      d.qpred = F.d_qpred;
      d.tiles = F.d_tiles;
      d.cap = (size_t)F.f->ngrid * F.f->ld;
      d.first = p.first_before[f];
      d.n = F.f->ngrid;
      d.ld = F.f->ld;
      d.nslice = r->nslice;
      d.harm = F.harm;
      d.do_source = st.in_undulator && (F.harm % 2) == 1 && p.fc[f] != 0.0;
      d.gridmax = (float)F.f->gridmax;
      d.dgrid = (float)F.f->dgrid;
      d.inv_dgrid = (float)(1.0 / F.f->dgrid);
      // adi_compute_slice_scl (src/Core/FieldSolverADICUDA.cpp:75-96)
      d.kscl = p.fc[f] * 376.73031346177 * F.f->xks * st.delz /
               (4.0 * 510998.95 * F.f->dgrid * F.f->dgrid);
      d.tile_cells = F.tile_cells;
    }
    L.dd = a;
  }
  // K3/K4 per field
  for (int f = 0; f < r->nfield; ++f) {
    RunFieldState& F = r->fs[f];
    F.f->first = p.first_before[f];
    const bool src = st.in_undulator && (F.harm % 2) == 1 && p.fc[f] != 0.0 && r->npart > 0;
    AdiYExtras ex{p.zero_start[f], p.zero_count[f], F.d_part};
    if (int rc = adi_plan(F.adis[p.adi_index[f]], F.f, src ? F.f->src : nullptr, F.f->desc, &ex,
                          L.adi[f]))
      return rc;
    F.f->first = p.first_after[f];
  }
  // K5
  {
    FinalizeArgs a{};
    a.nfield = r->nfield;
    a.nslice = r->nslice;
    a.field_hist = step_hist + r->rec_beam * r->nslice;
    for (int f = 0; f < r->nfield; ++f) {
      a.part[f] = r->fs[f].d_part;
      a.bbox[f] = r->fs[f].d_bbox;
      a.nband[f] = r->fs[f].nband;
      a.first_after[f] = p.first_after[f];
    }
    L.fa = a;
  }
  return G4B_OK;
}

// Launches one step of one run from its resolved arguments.
int launch_single(g4b_run* r, const StepArgs& L) {
  g4b_ctx* c = r->ctx;
  // every kernel of the step on the context's stream is a programmatic
  // dependent launch (launch_pdl): it starts while its predecessor drains
  if (L.has_beam) {
    LaunchScope ls(c, "run_beam_step");
    auto kern = r->nfield == 1 ? beam_step_kernel<1>
                               : (r->nfield == 2 ? beam_step_kernel<2> : beam_step_kernel<0>);
    G4B_CUDA_TRY(launch_pdl(kern, (unsigned)r->nchunk, kStepThreads, 0, c->stream, L.bs));
  }
  if (int rc = check_launch(c, "beam_step_kernel")) return rc;
  // The beam diagnostics depend only on K1: see dep_split.  The branch (beside
  // the deposition and the ADI passes, on SMs those leave idle, joined before
  // the finalize) is for large runs: a fork per step takes a graph long to
  // instantiate.
  const DepSplit sp = dep_split(r->nslice, (int)r->max_np, c->sm_count);
  const bool one = r->desc.nbunch == 1;
  const bool branch = r->nslice >= 2 * c->sm_count && r->capturing;
  if (branch) {
    G4B_CUDA_TRY(cudaEventRecord(r->ev_fork, c->stream));
    G4B_CUDA_TRY(cudaStreamWaitEvent(r->aux, r->ev_fork, 0));
    {
      LaunchScope ls(c, "run_beam_diag");
      (one ? beam_diag_kernel<1, false> : beam_diag_kernel<kMaxBunch, false>)<<<
          r->nslice, kDiagThreads, 0, r->aux>>>(L.bd);
    }
    if (int rc = check_launch(c, "beam_diag_kernel")) return rc;
    G4B_CUDA_TRY(cudaEventRecord(r->ev_join, r->aux));
  }
  if (sp.parts > 0) {
    LaunchScope ls(c, "run_deposit_diag");
    const DepDiagLaunch dl{L.dd, L.bd, sp.parts};
    G4B_CUDA_TRY(launch_pdl(dep_diag_kernel(one, sp), (unsigned)(r->nslice * sp.parts),
                            (unsigned)sp.T, sp.smem(), c->stream, dl));
  } else {
    LaunchScope ls(c, "run_deposit");
    G4B_CUDA_TRY(launch_pdl(branch ? deposit_kernel<false> : deposit_kernel<true>,
                            (unsigned)r->nslice, kDepThreads, dep_smem(kDepCells2), c->stream, L.dd));
  }
  if (int rc = check_launch(c, "deposit_kernel")) return rc;
  if (sp.parts == 0 && !branch) {
    {
      LaunchScope ls(c, "run_beam_diag");
      G4B_CUDA_TRY(launch_pdl(one ? beam_diag_kernel<1, true> : beam_diag_kernel<kMaxBunch, true>,
                              (unsigned)r->nslice, kDiagThreads, 0, c->stream, L.bd));
    }
    if (int rc = check_launch(c, "beam_diag_kernel")) return rc;
  }
  for (int f = 0; f < r->nfield; ++f)
    if (int rc = adi_launch(r->fs[f].f, L.adi[f])) return rc;
  if (branch) G4B_CUDA_TRY(cudaStreamWaitEvent(c->stream, r->ev_join, 0));
  {
    LaunchScope ls(c, "run_diag_finalize");
    G4B_CUDA_TRY(launch_pdl(diag_finalize_kernel,
                            (unsigned)((10 * r->nfield * r->nslice + 255) / 256), 256, 0,
                            c->stream, L.fa));
  }
  return check_launch(c, "diag_finalize_kernel");
}

int enqueue_step(g4b_run* r, int i, const StepPlan& p) {
  StepArgs L;
  if (int rc = build_step(r, i, p, L)) return rc;
  return launch_single(r, L);
}

std::vector<int> state_key(g4b_run* r) {
  std::vector<int> k;
  for (int f = 0; f < r->nfield; ++f) {
    k.push_back(r->fs[f].first);
    k.push_back(r->fs[f].f->mode);  // the ADI row layout the graph launches
    double a = r->fs[f].accuslip;
    int v[2];
    std::memcpy(v, &a, 8);
    k.push_back(v[0]);
    k.push_back(v[1]);
  }
  return k;
}

}  // namespace

extern "C" {

int g4b_run_create(g4b_ctx* c, const g4b_run_desc* d, const int64_t* off, g4b_run** out) {
  if (!d || !off || !out) return fail(G4B_ERR_ARG, "g4b_run_create: null arg");
  *out = nullptr;
  // The exact-integer deposition scales a slice's contributions so that the
  // fullest cell of its tile sums to at most 2^30; with at most kRunMaxNp
  // particles per slice every contribution keeps at least 2^30 / kRunMaxNp =
  // 2^14 quanta.  Checked before anything touches the device.
  if (d->nslice > 0)
    for (int s = 0; s < d->nslice; ++s)
      if (off[s + 1] - off[s] > kRunMaxNp)
        return fail(G4B_ERR_RANGE, "g4b_run_create: slice " + std::to_string(s) + " holds " +
                                       std::to_string(off[s + 1] - off[s]) +
                                       " particles; the mixed form takes at most " +
                                       std::to_string(kRunMaxNp) + " per slice");
  if (!c) return fail(G4B_ERR_ARG, "g4b_run_create: null ctx");
  if (d->nslice <= 0 || d->nfield < 1 || d->nfield > kRunFields || d->nbunch < 1 ||
      d->nbunch > kMaxBunch || !(d->gamma_ref > 1) || !(d->lambda0 > 0) || !(d->sample > 0))
    return fail(G4B_ERR_ARG, "g4b_run_create: bad descriptor");
  if (d->precision != G4B_MIXED)
    return fail(G4B_ERR_ARG, "g4b_run_create: the fused run holds mixed-precision state");
  for (int f = 0; f < d->nfield; ++f)
    if (d->ngrid[f] + 2 > kDepMaxWidth)
      return fail(G4B_ERR_ARG, "g4b_run_create: ngrid above the mixed form's limit (880)");
  if (off[0] != 0) return fail(G4B_ERR_ARG, "g4b_run_create: slice_offsets[0] != 0");
  G4B_CUDA_TRY(cudaSetDevice(c->device));
  auto r = new (std::nothrow) g4b_run();
  if (!r) return fail(G4B_ERR_NOMEM, "g4b_run_create: host allocation");
  r->ctx = c;
  ctx_retain(c);
  r->desc = *d;
  r->nslice = d->nslice;
  r->nfield = d->nfield;
  r->npart = off[d->nslice];
  std::vector<int4> chunks;
  for (int s = 0; s < d->nslice; ++s) {
    if (off[s + 1] < off[s]) {
      delete r;
      return fail(G4B_ERR_ARG, "g4b_run_create: slice offsets not monotonic");
    }
    r->max_np = std::max<int64_t>(r->max_np, off[s + 1] - off[s]);
    for (int64_t p = off[s]; p < off[s + 1]; p += kRunChunk) {
      const int64_t e = std::min<int64_t>(p + kRunChunk, off[s + 1]);
      chunks.push_back(make_int4(s, (int)(p & 0x7fffffff), (int)(e - p), (int)(p >> 31)));
    }
  }
  r->nchunk = (int)chunks.size();
  const size_t np = (size_t)std::max<int64_t>(r->npart, 1);
  cudaError_t e = cudaSuccess;
  auto A = [&](void** p, size_t b) {
    if (e == cudaSuccess) e = dev_alloc(c, p, b);
    if (e == cudaSuccess) r->bytes += b;
  };
  A((void**)&r->xy, np * 8);
  A((void**)&r->pxy, np * 8);
  A((void**)&r->dg, np * 4);
  A((void**)&r->th, np * 8);
  A((void**)&r->d_off, (d->nslice + 1) * 8);
  A((void**)&r->d_chunks, std::max(1, r->nchunk) * sizeof(int4));
  A((void**)&r->d_current, d->nslice * 8);
  A((void**)&r->d_eloss, d->nslice * 8);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(r->d_off, off, (d->nslice + 1) * 8, cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess && r->nchunk)
    e = cudaMemcpyAsync(r->d_chunks, chunks.data(), chunks.size() * sizeof(int4),
                        cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(r->d_current, 0, d->nslice * 8, c->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(r->d_eloss, 0, d->nslice * 8, c->stream);
  if (e != cudaSuccess) {
    g4b_run_destroy(r);
    return cuda_fail(e, "g4b_run_create: device allocation");
  }
  for (int f = 0; f < d->nfield; ++f) {
    RunFieldState& F = r->fs[f];
    F.harm = d->harm[f];
    int rc = g4b_field_create(c, d->nslice, d->ngrid[f], d->gridmax[f],
                              d->lambda0 / (double)d->harm[f], d->harm[f], G4B_MIXED, 0, &F.f);
    if (rc) {
      g4b_run_destroy(r);
      return rc;
    }
    r->bytes += F.f->bytes;
    F.nband = (F.f->ngrid + F.f->band_rows - 1) / F.f->band_rows;
    A((void**)&F.d_bbox, d->nslice * sizeof(int4));
    A((void**)&F.d_mpred, d->nslice * sizeof(int));
    A((void**)&F.d_qpred, d->nslice * sizeof(float));
    F.tile_cells = std::min((F.f->ngrid * F.f->ld + 3) / 4 * 4, kDepTileCells);
    const size_t tiles =
        dep_split_few(d->nslice, c->sm_count).parts > 0 ? d->nslice * dep_tile_bytes(F.tile_cells) : 0;
    if (tiles) A((void**)&F.d_tiles, tiles);
    A((void**)&F.d_part, (size_t)d->nslice * F.nband * 9 * 8);
    if (e != cudaSuccess) {
      g4b_run_destroy(r);
      return cuda_fail(e, "g4b_run_create: device allocation");
    }
    std::vector<int4> init(d->nslice, make_int4(1 << 30, 1 << 30, -1, -1));
    e = cudaMemcpyAsync(F.d_bbox, init.data(), init.size() * sizeof(int4),
                        cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess)
      e = cudaMemsetAsync(F.d_mpred, 0, d->nslice * sizeof(int), c->stream);
    if (e == cudaSuccess)
      e = cudaMemsetAsync(F.d_qpred, 0, d->nslice * sizeof(float), c->stream);
    if (e == cudaSuccess && tiles) e = cudaMemsetAsync(F.d_tiles, 0, tiles, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) {
      g4b_run_destroy(r);
      return cuda_fail(e, "g4b_run_create: bbox init");
    }
  }
  r->rec_beam = kBeamRec + 2 * d->nbunch;
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) {
    g4b_run_destroy(r);
    return cuda_fail(e, "g4b_run_create: device allocation");
  }
  r->step_doubles = (size_t)d->nslice * (r->rec_beam + 9 * d->nfield);
  for (const DepSplit s : {DepSplit{3, 512}, DepSplit{2, 512}, DepSplit{2, 256}})
    for (const bool one : {false, true})
      cudaFuncSetAttribute(dep_diag_kernel(one, s), cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)s.smem());
  cudaFuncSetAttribute(deposit_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)dep_smem(kDepCells2));
  cudaFuncSetAttribute(deposit_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)dep_smem(kDepCells2));
  *out = r;
  return G4B_OK;
}

int g4b_run_destroy(g4b_run* r) {
  if (!r) return G4B_OK;
  ctx_quiesce(r->ctx);
  if (r->gexec) cudaGraphExecDestroy(r->gexec);
  if (r->ev_fork) cudaEventDestroy(r->ev_fork);
  if (r->ev_join) cudaEventDestroy(r->ev_join);
  if (r->aux) cudaStreamDestroy(r->aux);
  void* ptrs[] = {r->xy, r->pxy, r->dg, r->th, r->d_off, r->d_chunks, r->d_current,
                  r->d_eloss, r->d_hist};
  for (void* p : ptrs) dev_free(r->ctx, p);
  for (int f = 0; f < kRunFields; ++f) {
    RunFieldState& F = r->fs[f];
    for (g4b_adi* a : F.adis) g4b_adi_destroy(a);
    if (F.f) g4b_field_destroy(F.f);
    dev_free(r->ctx, F.d_bbox);
    dev_free(r->ctx, F.d_mpred);
    dev_free(r->ctx, F.d_qpred);
    dev_free(r->ctx, F.d_tiles);
    dev_free(r->ctx, F.d_part);
  }
  ctx_release(r->ctx);
  delete r;
  return G4B_OK;
}

// FP64 particle arrays cross the bus and are converted on the device, in
// chunks through a staging buffer (theta stays FP64 and is copied directly).
int g4b_run_upload_beam(g4b_run* r, const double* x, const double* y, const double* px,
                        const double* py, const double* gamma, const double* theta) {
  if (!r || !x || !y || !px || !py || !gamma || !theta)
    return fail(G4B_ERR_ARG, "g4b_run_upload_beam: null arg");
  G4B_CUDA_TRY(cudaSetDevice(r->ctx->device));
  const size_t n = (size_t)r->npart;
  cudaStream_t s = r->ctx->stream;
  if (n == 0) return G4B_OK;
  const size_t chunk = std::min(n, (size_t)(64u << 20) / 40);
  double* stage = nullptr;
  G4B_CUDA_TRY(dev_alloc(r->ctx, (void**)&stage, chunk * 40));
  const double* src[5] = {x, y, px, py, gamma};
  cudaError_t e = cudaMemcpyAsync(r->th, theta, n * 8, cudaMemcpyHostToDevice, s);
  const float gf = (float)r->desc.gamma_ref;
  for (size_t p0 = 0; p0 < n && e == cudaSuccess; p0 += chunk) {
    const size_t m = std::min(chunk, n - p0);
    for (int k = 0; k < 5 && e == cudaSuccess; ++k)
      e = cudaMemcpyAsync(stage + k * chunk, src[k] + p0, m * 8, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
      const unsigned grid = (unsigned)std::min<size_t>((m + 255) / 256, 1u << 20);
      beam_f64_to_mixed<<<grid, 256, 0, s>>>(stage, chunk, m, gf, r->xy + p0, r->pxy + p0,
                                             r->dg + p0);
      e = cudaGetLastError();
    }
  }
  dev_free(r->ctx, stage);
  // a new beam: the next deposition counts before it accumulates
  for (int f = 0; f < r->nfield && e == cudaSuccess; ++f) {
    e = cudaMemsetAsync(r->fs[f].d_mpred, 0, r->nslice * sizeof(int), s);
    if (e == cudaSuccess)
      e = cudaMemsetAsync(r->fs[f].d_qpred, 0, r->nslice * sizeof(float), s);
  }
  const cudaError_t es = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_fail(e, "g4b_run_upload_beam");
  if (es != cudaSuccess) return cuda_fail(es, "g4b_run_upload_beam");
  return G4B_OK;
}

int g4b_run_download_beam(g4b_run* r, double* x, double* y, double* px, double* py,
                          double* gamma, double* theta) {
  if (!r) return fail(G4B_ERR_ARG, "g4b_run_download_beam: null run");
  G4B_CUDA_TRY(cudaSetDevice(r->ctx->device));
  const size_t n = (size_t)r->npart;
  cudaStream_t s = r->ctx->stream;
  if (n == 0) return read_device_error(r->ctx, "g4b_run_download_beam");
  const size_t chunk = std::min(n, (size_t)(64u << 20) / 40);
  double* stage = nullptr;
  G4B_CUDA_TRY(dev_alloc(r->ctx, (void**)&stage, chunk * 40));
  double* dst[5] = {x, y, px, py, gamma};
  cudaError_t e = theta ? cudaMemcpyAsync(theta, r->th, n * 8, cudaMemcpyDeviceToHost, s)
                        : cudaSuccess;
  const double gf = (double)(float)r->desc.gamma_ref;
  for (size_t p0 = 0; p0 < n && e == cudaSuccess; p0 += chunk) {
    const size_t m = std::min(chunk, n - p0);
    const unsigned grid = (unsigned)std::min<size_t>((m + 255) / 256, 1u << 20);
    beam_mixed_to_f64<<<grid, 256, 0, s>>>(r->xy + p0, r->pxy + p0, r->dg + p0, gf, m, stage,
                                           chunk);
    e = cudaGetLastError();
    for (int k = 0; k < 5 && e == cudaSuccess; ++k)
      if (dst[k]) e = cudaMemcpyAsync(dst[k] + p0, stage + k * chunk, m * 8,
                                      cudaMemcpyDeviceToHost, s);
  }
  dev_free(r->ctx, stage);
  const cudaError_t es = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_fail(e, "g4b_run_download_beam");
  if (es != cudaSuccess) return cuda_fail(es, "g4b_run_download_beam");
  return read_device_error(r->ctx, "g4b_run_download_beam");
}

int g4b_run_upload_field(g4b_run* r, int fi, const double* cells, int first) {
  if (!r || fi < 0 || fi >= r->nfield || first < 0 || first >= r->nslice)
    return fail(G4B_ERR_ARG, "g4b_run_upload_field: bad argument");
  RunFieldState& F = r->fs[fi];
  if (cells) {
    if (int rc = g4b_field_upload(F.f, cells)) return rc;
  } else {  // a zero field (no seed)
    G4B_CUDA_TRY(cudaSetDevice(r->ctx->device));
    G4B_CUDA_TRY(cudaMemsetAsync(F.f->a, 0, (size_t)F.f->nslice * F.f->ngrid * F.f->ld *
                                                F.f->cell_bytes, r->ctx->stream));
    G4B_CUDA_TRY(cudaStreamSynchronize(r->ctx->stream));
  }
  if (int rc = g4b_field_set_first(F.f, first)) return rc;
  F.first = first;
  F.accuslip = 0.0;
  return G4B_OK;
}

int g4b_run_download_field(g4b_run* r, int fi, double* cells, int* first) {
  if (!r || fi < 0 || fi >= r->nfield || !cells)
    return fail(G4B_ERR_ARG, "g4b_run_download_field: bad argument");
  RunFieldState& F = r->fs[fi];
  if (int rc = g4b_field_download(F.f, cells)) return rc;
  if (first) *first = F.first;
  return read_device_error(r->ctx, "g4b_run_download_field");
}

int g4b_run_set_current(g4b_run* r, const double* current) {
  if (!r || !current) return fail(G4B_ERR_ARG, "g4b_run_set_current: null arg");
  G4B_CUDA_TRY(cudaSetDevice(r->ctx->device));
  G4B_CUDA_TRY(cudaMemcpyAsync(r->d_current, current, r->nslice * 8, cudaMemcpyHostToDevice,
                               r->ctx->stream));
  G4B_CUDA_TRY(cudaStreamSynchronize(r->ctx->stream));
  return G4B_OK;
}

int g4b_run_set_eloss(g4b_run* r, const double* eloss) {
  if (!r) return fail(G4B_ERR_ARG, "g4b_run_set_eloss: null run");
  G4B_CUDA_TRY(cudaSetDevice(r->ctx->device));
  if (eloss)
    G4B_CUDA_TRY(cudaMemcpyAsync(r->d_eloss, eloss, r->nslice * 8, cudaMemcpyHostToDevice,
                                 r->ctx->stream));
  else
    G4B_CUDA_TRY(cudaMemsetAsync(r->d_eloss, 0, r->nslice * 8, r->ctx->stream));
  G4B_CUDA_TRY(cudaStreamSynchronize(r->ctx->stream));
  return G4B_OK;
}

int g4b_run_set_lattice(g4b_run* r, int nstep, const g4b_step* steps, const double* fc,
                        const double* slip, int hist_steps) {
  if (!r || nstep <= 0 || !steps || !fc || !slip)
    return fail(G4B_ERR_ARG, "g4b_run_set_lattice: bad argument");
  G4B_CUDA_TRY(cudaSetDevice(r->ctx->device));
  r->steps.assign(steps, steps + nstep);
  r->fc.assign(fc, fc + (size_t)nstep * r->nfield);
  r->slip.assign(slip, slip + nstep);
  // one FP64 factorisation per distinct step length and field grid
  for (int f = 0; f < r->nfield; ++f) {
    RunFieldState& F = r->fs[f];
    for (int i = 0; i < nstep; ++i) {
      const double dz = steps[i].delz;
      if (std::find(F.adi_delz.begin(), F.adi_delz.end(), dz) != F.adi_delz.end()) continue;
      g4b_adi* a = nullptr;
      if (int rc = g4b_adi_create(r->ctx, &a)) return rc;
      if (int rc = g4b_adi_init(a, dz, F.f->dgrid, F.f->xks, F.f->ngrid)) {
        g4b_adi_destroy(a);
        return rc;
      }
      F.adis.push_back(a);
      F.adi_delz.push_back(dz);
    }
    if (int rc = adi_configure(F.f)) return rc;
  }
  const int hs = hist_steps > 0 ? hist_steps : nstep;
  dev_free(r->ctx, r->d_hist);
  r->d_hist = nullptr;
  G4B_CUDA_TRY(dev_alloc(r->ctx, (void**)&r->d_hist, (size_t)hs * r->step_doubles * 8));
  G4B_CUDA_TRY(cudaMemsetAsync(r->d_hist, 0, (size_t)hs * r->step_doubles * 8, r->ctx->stream));
  r->hist_steps = hs;
  if (r->gexec) {
    cudaGraphExecDestroy(r->gexec);
    r->gexec = nullptr;
  }
  return G4B_OK;
}

static int run_capture(g4b_run* r, int first_step, int nsteps, cudaGraphExec_t* out) {
  g4b_ctx* c = r->ctx;
  cudaGraph_t g = nullptr;
  if (!r->aux) {
    G4B_CUDA_TRY(cudaStreamCreateWithFlags(&r->aux, cudaStreamNonBlocking));
    G4B_CUDA_TRY(cudaEventCreateWithFlags(&r->ev_fork, cudaEventDisableTiming));
    G4B_CUDA_TRY(cudaEventCreateWithFlags(&r->ev_join, cudaEventDisableTiming));
  }
  const bool prof = c->prof.on;  // no profiler events inside a graph
  c->prof.on = false;
  G4B_CUDA_TRY(cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
  r->capturing = true;
  int rc = G4B_OK;
  for (int k = 0; k < nsteps && rc == G4B_OK; ++k) {
    const int i = (first_step + k) % (int)r->steps.size();
    StepPlan p;
    rc = plan_step(r, i, p);
    if (rc == G4B_OK) rc = enqueue_step(r, first_step + k, p);
  }
  r->capturing = false;
  cudaError_t e = cudaStreamEndCapture(c->stream, &g);
  c->prof.on = prof;
  if (rc) {
    if (g) cudaGraphDestroy(g);
    return rc;
  }
  if (e != cudaSuccess) return cuda_fail(e, "cudaStreamEndCapture");
  e = cudaGraphInstantiate(out, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGraphInstantiate");
  return G4B_OK;
}

// Enqueue lattice steps [first_step, first_step + nsteps) (indices wrap).
// use_graph: 0 = direct launches; 1 = replay a CUDA graph of the whole
// range (captured on first use and reused while the range and the slippage
// state match).
static int run_capture(g4b_run* r, int first_step, int nsteps, cudaGraphExec_t* out);

static int run_prepare(g4b_run* r, int first_step, int nsteps) {
  std::vector<int> key = state_key(r);
  const bool hit = r->gexec && r->g_first == first_step && r->g_n == nsteps && r->g_state == key;
  if (hit) return G4B_OK;
  if (r->gexec) cudaGraphExecDestroy(r->gexec);
  r->gexec = nullptr;
  // capture advances the host slippage model; restore it afterwards
  int first[kRunFields];
  double acc[kRunFields];
  for (int f = 0; f < r->nfield; ++f) {
    first[f] = r->fs[f].first;
    acc[f] = r->fs[f].accuslip;
  }
  int rc = run_capture(r, first_step, nsteps, &r->gexec);
  for (int f = 0; f < r->nfield; ++f) {
    r->fs[f].first = first[f];
    r->fs[f].accuslip = acc[f];
    r->fs[f].f->first = first[f];
  }
  if (rc) return rc;
  r->g_first = first_step;
  r->g_n = nsteps;
  r->g_state = key;
  return G4B_OK;
}

// Capture (without launching) the CUDA graph of steps [first_step,
// first_step + nsteps) from the current state, for a later g4b_run_advance
// with use_graph on the same range.
int g4b_run_prepare(g4b_run* r, int first_step, int nsteps) {
  if (!r || nsteps <= 0 || first_step < 0) return fail(G4B_ERR_ARG, "g4b_run_prepare: bad arg");
  if (r->steps.empty()) return fail(G4B_ERR_STATE, "g4b_run_prepare: no lattice");
  G4B_CUDA_TRY(cudaSetDevice(r->ctx->device));
  return run_prepare(r, first_step, nsteps);
}

int g4b_run_advance(g4b_run* r, int first_step, int nsteps, int use_graph) {
  if (!r || nsteps < 0 || first_step < 0) return fail(G4B_ERR_ARG, "g4b_run_advance: bad arg");
  if (r->steps.empty()) return fail(G4B_ERR_STATE, "g4b_run_advance: no lattice");
  G4B_CUDA_TRY(cudaSetDevice(r->ctx->device));
  if (!use_graph) {
    for (int k = 0; k < nsteps; ++k) {
      const int i = (first_step + k) % (int)r->steps.size();
      StepPlan p;
      if (int rc = plan_step(r, i, p)) return rc;
      if (int rc = enqueue_step(r, first_step + k, p)) return rc;
    }
    return G4B_OK;
  }
  if (int rc = run_prepare(r, first_step, nsteps)) return rc;
  r->ctx->launches += (uint64_t)nsteps * (4 + 2 * r->nfield);
  G4B_CUDA_TRY(cudaGraphLaunch(r->gexec, r->ctx->stream));
  // advance the host model exactly as the captured steps did
  for (int k = 0; k < nsteps; ++k) {
    StepPlan p;
    if (int rc = plan_step(r, (first_step + k) % (int)r->steps.size(), p)) return rc;
    for (int f = 0; f < r->nfield; ++f) r->fs[f].f->first = p.first_after[f];
  }
  return G4B_OK;
}

// Diagnostics of lattice step `step` (the history keeps the last hist_steps
// steps): beam[nslice*(23+2*nbunch)] in the reference's stats order, field
// [nfield*nslice*9] = power, x1, x2, y1, y2, farfield re/im, centre re/im,
// indexed by beam slice.  Synchronises.
int g4b_run_history(g4b_run* r, int step, double* beam, double* field) {
  if (!r || step < 0) return fail(G4B_ERR_ARG, "g4b_run_history: bad arg");
  if (!r->d_hist) return fail(G4B_ERR_STATE, "g4b_run_history: no lattice");
  G4B_CUDA_TRY(cudaSetDevice(r->ctx->device));
  const double* h = r->d_hist + (size_t)(step % r->hist_steps) * r->step_doubles;
  const size_t nb = (size_t)r->nslice * r->rec_beam;
  if (beam)
    G4B_CUDA_TRY(cudaMemcpyAsync(beam, h, nb * 8, cudaMemcpyDeviceToHost, r->ctx->stream));
  if (field)
    G4B_CUDA_TRY(cudaMemcpyAsync(field, h + nb, (size_t)r->nfield * r->nslice * 9 * 8,
                                 cudaMemcpyDeviceToHost, r->ctx->stream));
  G4B_CUDA_TRY(cudaStreamSynchronize(r->ctx->stream));
  return read_device_error(r->ctx, "g4b_run_history");
}

// Diagnostics of steps [first, first + n) in one read: out[n][step record],
// a step record being beam [nslice][23 + 2 nbunch] then field [nfield][nslice][9].
int g4b_run_history_range(g4b_run* r, int first, int n, double* out) {
  if (!r || first < 0 || n < 0 || !out) return fail(G4B_ERR_ARG, "g4b_run_history_range: bad arg");
  if (!r->d_hist) return fail(G4B_ERR_STATE, "g4b_run_history_range: no lattice");
  if (n > r->hist_steps)
    return fail(G4B_ERR_RANGE, "g4b_run_history_range: more steps than the history keeps");
  G4B_CUDA_TRY(cudaSetDevice(r->ctx->device));
  const size_t sd = r->step_doubles;
  int done = 0;
  while (done < n) {
    const int slot = (first + done) % r->hist_steps;
    const int cnt = std::min(n - done, r->hist_steps - slot);
    G4B_CUDA_TRY(cudaMemcpyAsync(out + (size_t)done * sd, r->d_hist + (size_t)slot * sd,
                                 (size_t)cnt * sd * 8, cudaMemcpyDeviceToHost, r->ctx->stream));
    done += cnt;
  }
  G4B_CUDA_TRY(cudaStreamSynchronize(r->ctx->stream));
  return read_device_error(r->ctx, "g4b_run_history_range");
}

int g4b_run_device_bytes(g4b_run* r, uint64_t* bytes) {
  if (!r || !bytes) return fail(G4B_ERR_ARG, "g4b_run_device_bytes: null arg");
  *bytes = r->bytes + (uint64_t)r->hist_steps * r->step_doubles * 8;
  return G4B_OK;
}

}  // extern "C"

// =========================================================== batched runs ===
// Many independent runs advanced together: per step one persistent launch
// per kernel phase covers every attached run.  Each run keeps its own state
// (a g4b_run); the engine resolves every run's step arguments on the host
// (build_step, the same code the single-run path uses), uploads them with
// one copy, and the batch kernels walk work lists of (run, chunk / slice /
// band) items.  Every item is computed exactly as in the single-run kernels,
// so a run's results do not depend on what else is in the batch.

namespace {

// ADI kernel modes (pick_mode): 32-lane rows, then 16-lane rows
constexpr int kNumM = 22;
const int kMList[kNumM] = {1,   3,   5,   7,   9,   11,  13,  15,  17,  21,  25,
                           33,  105, 107, 109, 111, 113, 115, 117, 121, 125, 133};
int m_index(int M) {
  for (int i = 0; i < kNumM; ++i)
    if (kMList[i] == M) return i;
  return -1;
}

// counts block at the head of the staging area
struct BatchCounts {
  int beam, dep, fin, pad;
  int adi[kNumM];
};

template <typename T>
size_t align_up(size_t x) {
  const size_t a = alignof(T) < 128 ? 128 : alignof(T);
  return (x + a - 1) / a * a;
}

}  // namespace

struct g4b_batch {
  g4b_ctx* ctx = nullptr;
  int max_runs = 0;
  std::vector<g4b_run*> runs;   // per slot (nullptr = free)
  std::vector<int> next, last;  // per slot: next lattice step, end (exclusive)
  bool dirty = true;            // composition changed since the last upload
  // staging (pinned host, double-buffered) and device mirror
  size_t off_bs = 0, off_dd = 0, off_bd = 0, off_fa = 0, off_ax = 0, off_ay = 0, off_mx = 0, off_my = 0,
         args_bytes = 0;
  unsigned char* h_args[2] = {nullptr, nullptr};
  unsigned char* d_args = nullptr;
  cudaEvent_t copied[2] = {nullptr, nullptr};
  int buf = 0;
  // work lists
  std::vector<int2> beam_items, dep_items;
  std::vector<int4> adi_items[kNumM];
  std::vector<int> modes;       // ADI row layout each [slot][field] is listed under
  size_t items_cap = 0, h_items_cap[2] = {0, 0};
  unsigned char* d_items = nullptr;
  unsigned char* h_items[2] = {nullptr, nullptr};  // pinned, alternating
  cudaEvent_t items_copied[2] = {nullptr, nullptr};
  int ibuf = 0;
  int stable = 0;               // steps since the composition last changed
  size_t off_beam = 0, off_dep = 0, off_adi[kNumM] = {};
  BatchCounts counts{};
  size_t smem_x[kNumM] = {}, smem_y[kNumM] = {};
  // push kernel field count (1 or 2 when every run has it, else 0 = any:
  // the single-run kernel of the same count), deposition bunching kind
  int nf_kind = 1, nb_kind = 1;
  // launch shapes (CTAs per kernel), chosen by the tuner
  int grid[4] = {0, 0, 0, 0};    // beam, deposit, adi, finalize
  int tune_left = 0, tune_idx = 0;
  std::vector<float> tune_ms[4];

  cudaEvent_t ev[5] = {};
  // concurrent branches of a step: the beam diagnostics beside the
  // deposition and ADI passes; the ADI kernels of different row layouts
  // beside one another
  static constexpr int kAux = 12;
  cudaStream_t aux[kAux] = {};
  cudaEvent_t ev_fork[2] = {}, ev_diag = nullptr, ev_adi[kAux] = {};
  // graph of one step for the current composition and shapes
  cudaGraphExec_t gexec = nullptr;
  bool graph_valid = false;
  uint64_t steps_done = 0;
};

namespace {

// The tuner's candidates per kernel, in units of SMs.
const int kTuneBeam[4] = {4, 8, 16, 32};
const int kTuneDep[4] = {2, 4, 6, 8};
const int kTuneAdi[4] = {2, 4, 6, 8};
constexpr int kDepBatchCtas = 2;  // the untuned deposition's

// The first `n` branch streams (a batch of more row layouts than usual gets the
// others when it is listed).
int batch_streams(g4b_batch* b, int n) {
  for (int k = 0; k < std::min(n, g4b_batch::kAux); ++k)
    if (!b->aux[k]) G4B_CUDA_TRY(cudaStreamCreateWithFlags(&b->aux[k], cudaStreamNonBlocking));
  return G4B_OK;
}

int batch_layout(g4b_batch* b) {
  size_t o = align_up<BatchCounts>(sizeof(BatchCounts));
  const size_t nr = b->max_runs, nf = (size_t)b->max_runs * kRunFields;
  b->off_bs = o;
  o = align_up<BeamStepArgs>(o + nr * sizeof(BeamStepArgs));
  b->off_dd = o;
  o = align_up<DepArgs>(o + nr * sizeof(DepArgs));
  b->off_bd = o;
  o = align_up<BeamDiagArgs>(o + nr * sizeof(BeamDiagArgs));
  b->off_fa = o;
  o = align_up<FinalizeArgs>(o + nr * sizeof(FinalizeArgs));
  b->off_ax = o;
  o = align_up<AdiPassArgs>(o + nf * sizeof(AdiPassArgs));
  b->off_ay = o;
  o = align_up<AdiPassArgs>(o + nf * sizeof(AdiPassArgs));
  b->off_mx = o;
  o = align_up<CUtensorMap>(o + nf * sizeof(CUtensorMap));
  b->off_my = o;
  o = align_up<CUtensorMap>(o + nf * sizeof(CUtensorMap));
  b->args_bytes = o;
  for (int k = 0; k < 2; ++k) {
    G4B_CUDA_TRY(cudaMallocHost(&b->h_args[k], o));
    std::memset(b->h_args[k], 0, o);
    G4B_CUDA_TRY(cudaEventCreateWithFlags(&b->copied[k], cudaEventDisableTiming));
  }
  G4B_CUDA_TRY(cudaMalloc(&b->d_args, o));
  for (auto& e : b->ev) G4B_CUDA_TRY(cudaEventCreate(&e));
  for (auto& e : b->ev_fork) G4B_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  for (auto& e : b->ev_adi) G4B_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  G4B_CUDA_TRY(cudaEventCreateWithFlags(&b->ev_diag, cudaEventDisableTiming));
  return batch_streams(b, 4);
}

// Rebuild the work lists after the set of attached, unfinished runs changed.
int batch_rebuild(g4b_batch* b) {
  b->beam_items.clear();
  b->dep_items.clear();
  for (auto& v : b->adi_items) v.clear();
  std::memset(b->smem_x, 0, sizeof b->smem_x);
  std::memset(b->smem_y, 0, sizeof b->smem_y);
  b->nf_kind = -1;
  b->nb_kind = 1;
  int nactive = 0;
  for (int s = 0; s < b->max_runs; ++s) {
    g4b_run* r = b->runs[s];
    if (!r || b->next[s] >= b->last[s]) continue;
    ++nactive;
    const int kind = r->nfield <= 2 ? r->nfield : 0;
    if (b->nf_kind < 0) b->nf_kind = kind;
    else if (b->nf_kind != kind) b->nf_kind = 0;
    if (r->desc.nbunch != 1) b->nb_kind = 0;
    for (int k = 0; k < r->nchunk; ++k) b->beam_items.push_back(make_int2(s, k));
    for (int sl = 0; sl < r->nslice; ++sl) b->dep_items.push_back(make_int2(s, sl));
    for (int f = 0; f < r->nfield; ++f) {
      g4b_field* F = r->fs[f].f;
      const int mi = m_index(F->mode);
      b->modes[s * kRunFields + f] = F->mode;
      if (mi < 0) return fail(G4B_ERR_RANGE, "g4b_batch: unsupported grid");
      const int nband = (F->ngrid + F->band_rows - 1) / F->band_rows;
      for (int sl = 0; sl < r->nslice; ++sl)
        for (int bd = 0; bd < nband; ++bd)
          b->adi_items[mi].push_back(make_int4(s * kRunFields + f, sl, bd, 0));
      // shared memory of the largest band in this group
      const int W = F->band_rows, ld = F->ld;
      const size_t cb = F->cell_bytes;
      const size_t out_bytes = (size_t)F->store_nbox * F->store_box_rows * W * cb;
      const size_t tx = (size_t)((W + 2) * ld + W * ld) * cb, ty = (size_t)(W * ld) * cb;
      // pass X: the output staging tile overlays the input tile
      b->smem_x[mi] = std::max(b->smem_x[mi], std::max(tx, out_bytes));
      b->smem_y[mi] = std::max(b->smem_y[mi], (ty + 127) / 128 * 128 + out_bytes);
    }
  }
  b->counts = BatchCounts{};
  b->counts.beam = (int)b->beam_items.size();
  b->counts.dep = (int)b->dep_items.size();
  b->counts.fin = nactive;
  size_t need = 0;
  b->off_beam = 0;
  need = align_up<int2>(b->beam_items.size() * sizeof(int2));
  b->off_dep = need;
  need = align_up<int2>(need + b->dep_items.size() * sizeof(int2));
  for (int m = 0; m < kNumM; ++m) {
    b->counts.adi[m] = (int)b->adi_items[m].size();
    b->off_adi[m] = need;
    need = align_up<int4>(need + b->adi_items[m].size() * sizeof(int4));
  }
  int ngroups = 0;
  for (int m = 0; m < kNumM; ++m) ngroups += b->counts.adi[m] > 0;
  if (int rc = batch_streams(b, ngroups)) return rc;
  need = std::max<size_t>(need, 256);
  if (need > b->items_cap) {  // stream-ordered: the old lists' readers finish first
    dev_free(b->ctx, b->d_items);
    b->d_items = nullptr;
    b->items_cap = 0;
    G4B_CUDA_TRY(dev_alloc(b->ctx, (void**)&b->d_items, need * 2));
    b->items_cap = need * 2;
  }
  // pinned staging, alternating buffers: wait only for the copy that used
  // this buffer two rebuilds ago
  const int k = b->ibuf;
  if (!b->items_copied[k])
    G4B_CUDA_TRY(cudaEventCreateWithFlags(&b->items_copied[k], cudaEventDisableTiming));
  G4B_CUDA_TRY(cudaEventSynchronize(b->items_copied[k]));
  if (need > b->h_items_cap[k]) {
    if (b->h_items[k]) cudaFreeHost(b->h_items[k]);
    b->h_items[k] = nullptr;
    b->h_items_cap[k] = 0;
    G4B_CUDA_TRY(cudaMallocHost(&b->h_items[k], need * 2));
    b->h_items_cap[k] = need * 2;
  }
  unsigned char* h = b->h_items[k];
  std::memcpy(h + b->off_beam, b->beam_items.data(), b->beam_items.size() * sizeof(int2));
  std::memcpy(h + b->off_dep, b->dep_items.data(), b->dep_items.size() * sizeof(int2));
  for (int m = 0; m < kNumM; ++m)
    std::memcpy(h + b->off_adi[m], b->adi_items[m].data(),
                b->adi_items[m].size() * sizeof(int4));
  G4B_CUDA_TRY(cudaMemcpyAsync(b->d_items, h, need, cudaMemcpyHostToDevice, b->ctx->stream));
  G4B_CUDA_TRY(cudaEventRecord(b->items_copied[k], b->ctx->stream));
  b->ibuf ^= 1;
  b->stable = 0;
  b->dirty = false;
  b->graph_valid = false;
  return G4B_OK;
}

// Has g4b_run_set_layouts switched a listed run's row layout since the last
// rebuild?  Its bands are then listed under another kernel than the one that
// its tables, which batch_stage takes from the layout in force, belong to.
bool batch_layouts_changed(const g4b_batch* b) {
  for (int s = 0; s < b->max_runs; ++s) {
    const g4b_run* r = b->runs[s];
    if (!r || b->next[s] >= b->last[s]) continue;
    for (int f = 0; f < r->nfield; ++f)
      if (r->fs[f].f->mode != b->modes[s * kRunFields + f]) return true;
  }
  return false;
}

// Resolve this step's arguments of every active run into the staging buffer.
int batch_stage(g4b_batch* b) {
  const int k = b->buf;
  G4B_CUDA_TRY(cudaEventSynchronize(b->copied[k]));  // the copy of two steps ago
  unsigned char* h = b->h_args[k];
  std::memcpy(h, &b->counts, sizeof(BatchCounts));
  auto* bs = reinterpret_cast<BeamStepArgs*>(h + b->off_bs);
  auto* dd = reinterpret_cast<DepArgs*>(h + b->off_dd);
  auto* bd = reinterpret_cast<BeamDiagArgs*>(h + b->off_bd);
  auto* fa = reinterpret_cast<FinalizeArgs*>(h + b->off_fa);
  auto* ax = reinterpret_cast<AdiPassArgs*>(h + b->off_ax);
  auto* ay = reinterpret_cast<AdiPassArgs*>(h + b->off_ay);
  auto* mx = reinterpret_cast<CUtensorMap*>(h + b->off_mx);
  auto* my = reinterpret_cast<CUtensorMap*>(h + b->off_my);
  int nfin = 0;
  for (int s = 0; s < b->max_runs; ++s) {
    g4b_run* r = b->runs[s];
    if (!r || b->next[s] >= b->last[s]) continue;
    const int i = b->next[s];
    StepPlan p;
    if (int rc = plan_step(r, i % (int)r->steps.size(), p)) return rc;
    StepArgs L;
    if (int rc = build_step(r, i, p, L)) return rc;
    bs[s] = L.bs;
    dd[s] = L.dd;
    bd[s] = L.bd;
    fa[nfin++] = L.fa;
    for (int f = 0; f < r->nfield; ++f) {
      ax[s * kRunFields + f] = L.adi[f].x;
      ay[s * kRunFields + f] = L.adi[f].y;
      mx[s * kRunFields + f] = *L.adi[f].tm_x;
      my[s * kRunFields + f] = *L.adi[f].tm_y;
    }
    b->next[s] = i + 1;
    if (b->next[s] >= b->last[s]) b->dirty = true;  // leaves the lists next step
  }
  G4B_CUDA_TRY(cudaMemcpyAsync(b->d_args, h, b->args_bytes, cudaMemcpyHostToDevice,
                               b->ctx->stream));
  G4B_CUDA_TRY(cudaEventRecord(b->copied[k], b->ctx->stream));
  b->buf ^= 1;
  return G4B_OK;
}

// The kernels of one batch step (capturable: no host synchronisation).
int batch_launch(g4b_batch* b, bool timed) {
  g4b_ctx* c = b->ctx;
  const int* counts = reinterpret_cast<const int*>(b->d_args);
  auto ev = [&](int i) {
    if (timed) cudaEventRecord(b->ev[i], c->stream);
  };
  ev(0);
  if (b->counts.beam > 0) {
    BeamBatchArgs a{reinterpret_cast<const BeamStepArgs*>(b->d_args + b->off_bs),
                    reinterpret_cast<const int2*>(b->d_items + b->off_beam), counts + 0};
    LaunchScope ls(c, "batch_beam_step");
    if (b->nf_kind == 1)
      beam_batch_kernel<1><<<b->grid[0], kStepThreads, 0, c->stream>>>(a);
    else if (b->nf_kind == 2)
      beam_batch_kernel<2><<<b->grid[0], kStepThreads, 0, c->stream>>>(a);
    else
      beam_batch_kernel<0><<<b->grid[0], kStepThreads, 0, c->stream>>>(a);
  }
  if (int rc = check_launch(c, "beam_batch_kernel")) return rc;
  ev(1);
  // several CTAs per slice, the diagnostics beside them, up to four slices per SM
  const DepSplit sp = dep_split_batch(b->counts.dep, c->sm_count);
  {
    DepBatchArgs a{reinterpret_cast<const DepArgs*>(b->d_args + b->off_dd),
                   reinterpret_cast<const int2*>(b->d_items + b->off_dep), counts + 1};
    LaunchScope ls(c, "batch_deposit");
    if (sp.parts > 0)
      dep_diag_batch_kernel(b->nb_kind == 1, sp)<<<b->counts.dep * sp.parts, sp.T, sp.smem(),
                                                   c->stream>>>(
          a, reinterpret_cast<const BeamDiagArgs*>(b->d_args + b->off_bd), sp.parts);
    else
      deposit_batch_kernel<<<b->grid[1], kDepThreads, dep_smem(kDepCells2), c->stream>>>(a);
  }
  if (int rc = check_launch(c, "deposit_batch_kernel")) return rc;
  // branches (not while the tuner or the profiler times single kernels)
  const bool fork = !timed && !c->prof.on;
  const DiagBatchArgs da{reinterpret_cast<const BeamDiagArgs*>(b->d_args + b->off_bd),
                         reinterpret_cast<const int2*>(b->d_items + b->off_dep), counts + 1};
  auto diag = [&](cudaStream_t st) {
    LaunchScope ls(c, "batch_beam_diag");
    if (b->nb_kind == 1)
      beam_diag_batch_kernel<1><<<2 * c->sm_count, kDiagThreads, 0, st>>>(da);
    else
      beam_diag_batch_kernel<kMaxBunch><<<2 * c->sm_count, kDiagThreads, 0, st>>>(da);
    return check_launch(c, "beam_diag_batch_kernel");
  };
  if (sp.parts > 0) {
    // computed beside the deposition
  } else if (fork) {
    G4B_CUDA_TRY(cudaEventRecord(b->ev_fork[0], c->stream));
    G4B_CUDA_TRY(cudaStreamWaitEvent(b->aux[0], b->ev_fork[0], 0));
    if (int rc = diag(b->aux[0])) return rc;
    G4B_CUDA_TRY(cudaEventRecord(b->ev_diag, b->aux[0]));
  } else if (int rc = diag(c->stream)) {
    return rc;
  }
  ev(2);
  auto adi = [&](cudaStream_t st, int m, int pass) {
    AdiBatchArgs a;
    a.args = reinterpret_cast<const AdiPassArgs*>(b->d_args + (pass ? b->off_ay : b->off_ax));
    a.maps = reinterpret_cast<const CUtensorMap*>(b->d_args + (pass ? b->off_my : b->off_mx));
    a.items = reinterpret_cast<const int4*>(b->d_items + b->off_adi[m]);
    a.nitems = reinterpret_cast<const int*>(b->d_args) + 4 + m;
    return adi_batch_launch(c, st, kMList[m], pass == 0, a, pass ? b->smem_y[m] : b->smem_x[m],
                            std::min(b->grid[2], b->counts.adi[m]));
  };
  int groups[kNumM], ngroups = 0;
  for (int m = 0; m < kNumM; ++m)
    if (b->counts.adi[m] > 0) groups[ngroups++] = m;
  if (fork && ngroups > 1) {
    // A group's pass Y waits for its own pass X alone: chains, round-robin over
    // the main stream and the branch streams 1..kAux-1 (stream 0 of the
    // branches carries the diagnostics).  A group of a few slices is bound by
    // its rows' latency, so chains gain by running at once: us per step of 32
    // runs of 9 row layouts, pass by pass over 4 streams 128, chains over 4
    // streams 124, over 6 122, a stream each 117.
    G4B_CUDA_TRY(cudaEventRecord(b->ev_fork[1], c->stream));
    for (int gi = 0; gi < ngroups; ++gi) {
      const int k = gi % g4b_batch::kAux;
      cudaStream_t st = k ? b->aux[k] : c->stream;
      if (k && gi == k) G4B_CUDA_TRY(cudaStreamWaitEvent(st, b->ev_fork[1], 0));
      for (int pass = 0; pass < 2; ++pass)
        if (int rc = adi(st, groups[gi], pass)) return rc;
    }
    for (int k = 1; k < std::min(ngroups, g4b_batch::kAux); ++k) {
      G4B_CUDA_TRY(cudaEventRecord(b->ev_adi[k], b->aux[k]));
      G4B_CUDA_TRY(cudaStreamWaitEvent(c->stream, b->ev_adi[k], 0));
    }
  } else {
    for (int pass = 0; pass < 2; ++pass) {
      for (int gi = 0; gi < ngroups; ++gi)
        if (int rc = adi(c->stream, groups[gi], pass)) return rc;
      ev(3 + pass);
    }
  }
  if (fork && sp.parts == 0) G4B_CUDA_TRY(cudaStreamWaitEvent(c->stream, b->ev_diag, 0));
  {
    LaunchScope ls(c, "batch_diag_finalize");
    finalize_batch_kernel<<<b->grid[3], 256, 0, c->stream>>>(
        reinterpret_cast<const FinalizeArgs*>(b->d_args + b->off_fa), counts + 2);
  }
  return check_launch(c, "finalize_batch_kernel");
}

void batch_default_grids(g4b_batch* b) {
  const int sm = b->ctx->sm_count;
  b->grid[0] = 2 * kStepBlocks * sm;
  b->grid[1] = kDepBatchCtas * sm;
  b->grid[2] = 4 * sm;
  b->grid[3] = sm;
}

}  // namespace

extern "C" {

int g4b_batch_create(g4b_ctx* c, int max_runs, g4b_batch** out) {
  if (!c || !out || max_runs < 1) return fail(G4B_ERR_ARG, "g4b_batch_create: bad arg");
  *out = nullptr;
  G4B_CUDA_TRY(cudaSetDevice(c->device));
  auto b = new (std::nothrow) g4b_batch();
  if (!b) return fail(G4B_ERR_NOMEM, "g4b_batch_create: host allocation");
  b->ctx = c;
  ctx_retain(c);
  b->max_runs = max_runs;
  b->runs.assign(max_runs, nullptr);
  b->next.assign(max_runs, 0);
  b->last.assign(max_runs, 0);
  b->modes.assign((size_t)max_runs * kRunFields, 0);
  batch_default_grids(b);
  cudaFuncSetAttribute(deposit_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)dep_smem(kDepCells2));
  for (const DepSplit s : {DepSplit{3, 512}, DepSplit{2, 512}})
    for (const bool one : {false, true})
      cudaFuncSetAttribute(dep_diag_batch_kernel(one, s),
                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.smem());
  if (int rc = batch_layout(b)) {
    g4b_batch_destroy(b);
    return rc;
  }
  *out = b;
  return G4B_OK;
}

int g4b_batch_destroy(g4b_batch* b) {
  if (!b) return G4B_OK;
  ctx_quiesce(b->ctx);
  if (b->gexec) cudaGraphExecDestroy(b->gexec);
  for (int k = 0; k < 2; ++k) {
    if (b->h_args[k]) cudaFreeHost(b->h_args[k]);
    if (b->copied[k]) cudaEventDestroy(b->copied[k]);
  }
  for (auto e : b->ev)
    if (e) cudaEventDestroy(e);
  for (auto e : b->ev_fork)
    if (e) cudaEventDestroy(e);
  for (auto e : b->ev_adi)
    if (e) cudaEventDestroy(e);
  if (b->ev_diag) cudaEventDestroy(b->ev_diag);
  for (auto s : b->aux)
    if (s) cudaStreamDestroy(s);
  if (b->d_args) cudaFree(b->d_args);
  dev_free(b->ctx, b->d_items);
  for (int k = 0; k < 2; ++k) {
    if (b->h_items[k]) cudaFreeHost(b->h_items[k]);
    if (b->items_copied[k]) cudaEventDestroy(b->items_copied[k]);
  }
  ctx_release(b->ctx);
  delete b;
  return G4B_OK;
}

// Attach a prepared run (created, uploaded, lattice set): it takes part in
// the batch's steps from lattice step `first_step` for `nsteps` steps.
int g4b_batch_attach(g4b_batch* b, g4b_run* r, int first_step, int nsteps, int* slot) {
  if (!b || !r || !slot || nsteps < 0 || first_step < 0)
    return fail(G4B_ERR_ARG, "g4b_batch_attach: bad arg");
  if (r->ctx->device != b->ctx->device)
    return fail(G4B_ERR_ARG, "g4b_batch_attach: run on another device");
  if (r->steps.empty()) return fail(G4B_ERR_STATE, "g4b_batch_attach: run has no lattice");
  for (int f = 0; f < r->nfield; ++f)
    if (r->fs[f].f->precision != G4B_MIXED)
      return fail(G4B_ERR_ARG, "g4b_batch_attach: mixed-precision runs only");
  for (int s = 0; s < b->max_runs; ++s)
    if (b->runs[s] == r) return fail(G4B_ERR_STATE, "g4b_batch_attach: run already attached");
  for (int s = 0; s < b->max_runs; ++s) {
    if (b->runs[s]) continue;
    b->runs[s] = r;
    b->next[s] = first_step;
    b->last[s] = first_step + nsteps;
    b->dirty = true;
    *slot = s;
    return G4B_OK;
  }
  return fail(G4B_ERR_RANGE, "g4b_batch_attach: no free slot");
}

// Detach the run in `slot` (the run itself is not destroyed); later steps
// leave it out.  Steps already enqueued may still use it: destroy it only
// after they completed (a g4b_ctx_mark after its last step).
int g4b_batch_detach(g4b_batch* b, int slot) {
  if (!b || slot < 0 || slot >= b->max_runs || !b->runs[slot])
    return fail(G4B_ERR_ARG, "g4b_batch_detach: bad slot");
  b->runs[slot] = nullptr;
  b->dirty = true;
  return G4B_OK;
}

int g4b_batch_status(g4b_batch* b, int slot, int* next_step, int* remaining) {
  if (!b || slot < 0 || slot >= b->max_runs || !b->runs[slot])
    return fail(G4B_ERR_ARG, "g4b_batch_status: bad slot");
  if (next_step) *next_step = b->next[slot];
  if (remaining) *remaining = std::max(0, b->last[slot] - b->next[slot]);
  return G4B_OK;
}

// Start the tuner: the next 4 batch steps run with candidate launch shapes
// (per kernel: CTAs per SM) and time each kernel; the fastest shape of every
// kernel is kept.  Results do not depend on the shapes.
int g4b_batch_tune(g4b_batch* b) {
  if (!b) return fail(G4B_ERR_ARG, "g4b_batch_tune: null batch");
  b->tune_left = 4;
  b->tune_idx = 0;
  for (auto& v : b->tune_ms) v.assign(4, 0.f);
  return G4B_OK;
}

// The ADI row layouts, then the launch shapes as g4b_batch_tune.  For every
// grid size among the attached runs' fields that has two row layouts (32
// lanes of M elements, 16 lanes of M' elements) and at least
// kTuneRowsMinSlices slices in the batch, both passes are timed in each
// layout on a scratch field of that grid (its slice count up to 128, zeros,
// best of three launches after one untimed), before any step: the runs'
// state never advances in a trial layout, so every step of the batch uses
// the chosen layouts and equals an alone run given the same layouts.
constexpr int kTuneRowsMinSlices = 32;

int g4b_batch_tune_layouts(g4b_batch* b) {
  if (!b) return fail(G4B_ERR_ARG, "g4b_batch_tune_layouts: null batch");
  g4b_ctx* c = b->ctx;
  G4B_CUDA_TRY(cudaSetDevice(c->device));
  struct Group {
    int n = 0, nslice = 0;
    double gridmax = 0, xlambda = 0, delz = 0;
    std::vector<g4b_field*> fields;
  };
  std::vector<Group> groups;
  for (int s = 0; s < b->max_runs; ++s) {
    g4b_run* r = b->runs[s];
    if (!r || b->next[s] >= b->last[s] || r->steps.empty()) continue;
    for (int f = 0; f < r->nfield; ++f) {
      g4b_field* F = r->fs[f].f;
      if (!alt_mode(F->ngrid)) continue;
      Group* g = nullptr;
      for (auto& x : groups)
        if (x.n == F->ngrid) g = &x;
      if (!g) {
        groups.emplace_back();
        g = &groups.back();
        g->n = F->ngrid;
        g->gridmax = F->gridmax;
        g->xlambda = F->xlambda;
        g->delz = r->steps[0].delz > 0 ? r->steps[0].delz : 0.015;
      }
      g->nslice += F->nslice;
      g->fields.push_back(F);
    }
  }
  for (Group& g : groups) {
    // a grid with few slices in the batch keeps its default: its passes are
    // launch-bound, and a switch would add a row-layout group (two more
    // launches per step) to the batch
    if (g.nslice < kTuneRowsMinSlices) continue;
    g4b_field* f = nullptr;
    g4b_adi* adi = nullptr;
    int rc = g4b_field_create(c, std::min(g.nslice, 128), g.n, g.gridmax, g.xlambda, 1,
                              G4B_MIXED, 0, &f);
    if (rc == G4B_OK) rc = g4b_adi_create(c, &adi);
    if (rc == G4B_OK) rc = g4b_adi_init(adi, g.delz, f->dgrid, f->xks, g.n);
    const int modes[2] = {pick_mode(g.n, G4B_MIXED), alt_mode(g.n)};
    float best[2] = {1e30f, 1e30f};
    for (int k = 0; k < 2 && rc == G4B_OK; ++k) {
      rc = field_set_layout(f, modes[k]);
      AdiPlan P;
      if (rc == G4B_OK) rc = adi_plan(adi, f, nullptr, f->desc, nullptr, P);
      for (int it = 0; it < 4 && rc == G4B_OK; ++it) {
        cudaEventRecord(b->ev[0], c->stream);
        rc = adi_launch(f, P);
        cudaEventRecord(b->ev[1], c->stream);
        if (rc == G4B_OK) {
          cudaError_t e = cudaEventSynchronize(b->ev[1]);
          if (e != cudaSuccess) rc = cuda_fail(e, "g4b_batch_tune_layouts");
        }
        float ms = 0.f;
        cudaEventElapsedTime(&ms, b->ev[0], b->ev[1]);
        if (it > 0) best[k] = std::min(best[k], ms);
      }
    }
    if (rc == G4B_OK) rc = read_device_error(c, "g4b_batch_tune_layouts");
    g4b_adi_destroy(adi);
    g4b_field_destroy(f);
    if (rc != G4B_OK) return rc;
    const int pick = best[1] < best[0] ? modes[1] : modes[0];
    for (g4b_field* F : g.fields)
      if (int r2 = field_set_layout(F, pick)) return r2;
  }
  b->dirty = true;
  b->graph_valid = false;
  return g4b_batch_tune(b);
}
int g4b_default_layout(int ngrid) { return pick_mode(ngrid, G4B_MIXED); }

// ADI row layouts of a run's fields: M elements per lane on 32-lane rows, or
// 100 + M on 16-lane rows (two rows per warp).
int g4b_run_get_layouts(g4b_run* r, int* modes) {
  if (!r || !modes) return fail(G4B_ERR_ARG, "g4b_run_get_layouts: null arg");
  for (int f = 0; f < r->nfield; ++f) modes[f] = r->fs[f].f->mode;
  return G4B_OK;
}

// Sets them (each the default or the other layout of the field's grid), e.g.
// to rerun a batch-tuned run alone with the same FP32 rounding.
int g4b_run_set_layouts(g4b_run* r, const int* modes) {
  if (!r || !modes) return fail(G4B_ERR_ARG, "g4b_run_set_layouts: null arg");
  G4B_CUDA_TRY(cudaSetDevice(r->ctx->device));
  for (int f = 0; f < r->nfield; ++f)
    if (int rc = field_set_layout(r->fs[f].f, modes[f])) return rc;
  return G4B_OK;
}

// Launch shapes in use: CTAs of the beam, deposition, ADI and finalize kernels.
int g4b_batch_shapes(g4b_batch* b, int* grids) {
  if (!b || !grids) return fail(G4B_ERR_ARG, "g4b_batch_shapes: null arg");
  for (int k = 0; k < 4; ++k) grids[k] = b->grid[k];
  return G4B_OK;
}

// Advance every attached, unfinished run by `nsteps` lattice steps (runs that
// reach their end drop out).  With use_graph the kernels of a step are
// replayed from a CUDA graph captured for the current composition.
int g4b_batch_step(g4b_batch* b, int nsteps, int use_graph) {
  if (!b || nsteps < 0) return fail(G4B_ERR_ARG, "g4b_batch_step: bad arg");
  g4b_ctx* c = b->ctx;
  G4B_CUDA_TRY(cudaSetDevice(c->device));
  for (int k = 0; k < nsteps; ++k) {
    if (b->dirty || batch_layouts_changed(b))
      if (int rc = batch_rebuild(b)) return rc;
    if (b->counts.fin == 0) return G4B_OK;
    if (int rc = batch_stage(b)) return rc;
    if (b->tune_left > 0) {
      const int sm = c->sm_count, t = b->tune_idx;
      b->grid[0] = kTuneBeam[t] * sm;
      b->grid[1] = kTuneDep[t] * sm;
      b->grid[2] = kTuneAdi[t] * sm;
      if (int rc = batch_launch(b, true)) return rc;
      G4B_CUDA_TRY(cudaEventSynchronize(b->ev[4]));
      for (int q = 0; q < 3; ++q) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, b->ev[q], b->ev[q + 1]);
        b->tune_ms[q][t] = ms;
      }
      {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, b->ev[3], b->ev[4]);
        b->tune_ms[2][t] += ms;  // both ADI passes
      }
      b->tune_idx++;
      if (--b->tune_left == 0) {
        const int* cand[3] = {kTuneBeam, kTuneDep, kTuneAdi};
        // a deposition split over several CTAs per slice takes no notice of its
        // grid: the default stays for a later composition
        const bool split = dep_split_batch(b->counts.dep, sm).parts > 0;
        for (int q = 0; q < 3; ++q) {
          if (q == 1 && split) {
            b->grid[1] = kDepBatchCtas * sm;
            continue;
          }
          int best = 0;
          for (int j = 1; j < 4; ++j)
            if (b->tune_ms[q][j] < b->tune_ms[q][best]) best = j;
          b->grid[q] = cand[q][best] * sm;
        }
        b->graph_valid = false;
      }
    } else if (use_graph && b->stable >= 2) {
      // a graph pays once the composition holds for a few steps
      if (!b->graph_valid) {
        if (b->gexec) cudaGraphExecDestroy(b->gexec);
        b->gexec = nullptr;
        cudaGraph_t g;
        const bool prof = c->prof.on;  // no profiler events inside a graph
        c->prof.on = false;
        G4B_CUDA_TRY(cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
        const int rc = batch_launch(b, false);
        cudaError_t e = cudaStreamEndCapture(c->stream, &g);
        c->prof.on = prof;
        if (rc) return rc;
        if (e != cudaSuccess) return cuda_fail(e, "g4b_batch_step: capture");
        e = cudaGraphInstantiate(&b->gexec, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) return cuda_fail(e, "g4b_batch_step: instantiate");
        b->graph_valid = true;
      }
      G4B_CUDA_TRY(cudaGraphLaunch(b->gexec, c->stream));
    } else {
      if (int rc = batch_launch(b, false)) return rc;
    }
    b->steps_done++;
    b->stable++;
  }
  return G4B_OK;
}

}  // extern "C"
