// Near field of the complex Helmholtz kernel e^{ikr} / r and of the Yukawa
// kernel e^{-kr} / r (complex charges q, the 1/(4 pi) on output).
//
// Pairs at zero distance contribute nothing when the plan excludes them or
// when there is no softening; eps2 (the plan's softening) is added to r^2.
// Mixed form: FP32 terms, the hardware's sine and cosine of the phase (reduced
// to [-pi, pi] where it can exceed pi), summed over 32 sources in FP32, then
// in FP64.  FP64 form: everything in FP64 after the FP32 coordinates.
//
// Layout (as p2p_mixed.cu's): a block of 4 warps per work item of up to 128
// targets of a leaf, the neighbour leaves' sources staged as one list in chunks
// (p2p_list.cuh); a warp is 8 target lanes x 4 source streams, a lane holding
// NT <= 4 targets, so that a leaf of any size fills the lanes and a
// shared-memory read of sources serves NT targets; only the own leaf's runs and
// the last one, which can hold padding, test for zero distance.  (Mixed form: a chunk
// with a coordinate so close to zero that r^2 may be below FP32's normal range takes
// a plainer loop, near_zero_runs.)
//
// Bounds.  Mixed: the special-function pipe (rsqrt, sine and cosine: 3 of 16
// lanes a clock per pair, 3.57 G pairs in 2.3 ms), with the FP32 work next to it
// in the two-lane instructions (15 lane operations a pair).  FP64 form: the FP64
// pipe (50 operations a pair, 30 of them sine and cosine), the inverse root a
// hardware estimate and one third-order step.
//
// Measured against one or two targets a thread and scalar FP32 (or the library's
// square root and divisions), this phase alone on one B200: mixed, 1,048,576
// sphere points, k = 5, depth 5 (3.57 G pairs) 4.65 -> 2.75 ms; FP64, 30,011
// points, depth 3 (46.8 M pairs, 272 leaves) 1.41 -> 0.27 ms (0.38 with the
// library's sincos, whose branch keeps a lane's targets one after another).
#include <cuda_runtime.h>

#include <cmath>

#include "internal.h"
#include "kernels.h"
#include "p2p_list.cuh"

namespace fmmb {
namespace {

constexpr int kItem = 128;  // targets of a work item
// Warps of a block: 4; in the FP64 form 8 where all items are resident at once with 4
// (as p2p_f64.cu).  Whole evaluate with 4 / 8, us, p = 8: 64 points a leaf, 216 items
// 221 / 177, 512 385 / 360, 729 496 / 505, 1,331 899 / 899, 4,096 2,822 / 2,881; 110 a
// leaf, 216 items 458 / 366, 512 897 / 703, 729 1,016 / 993, 1,000 1,355 / 1,373, 4,096
// 5,824 / 5,972.
constexpr int kFewItems = 4 * 148;
constexpr int max_warps(bool f32) { return f32 ? 4 : 8; }
constexpr int kG = 8;        // targets of a group (lanes g = lane % 8)
constexpr int kS = 32 / kG;  // source streams of a warp (s = lane / 8)
constexpr int kMaxNT = 4;    // groups of a tile
constexpr int kCap = 512;    // staged sources per chunk (multiple of 32 * 4)

__device__ __forceinline__ float2 dup(float v) { return make_float2(v, v); }
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// F32: sources j, j + 1 (even j) packed for the two-lane FP32 instructions,
// (-x_j, -x_j+1, -y_j, -y_j+1), (-z_j, -z_j+1, Re q_j, Re q_j+1), (Im q_j, Im q_j+1).
// FP64: (x, y), (z, Re q), Im q.
template <bool F32>
struct Smem;
template <>
struct Smem<true> {
  float4 A[kCap / 2], B[kCap / 2];
  float2 Q[kCap / 2];
  double red[max_warps(true) - 1][kMaxNT][2][kG];
  SrcList src;
};
template <>
struct Smem<false> {
  double2 A[kCap], B[kCap];
  double Q[kCap];
  double red[max_warps(false) - 1][kMaxNT][2][kG];
  SrcList src;
};

// the lane's 4 source pairs of a run of 32 (pairs pb, pb + 4, ...) against its NT targets
template <bool YUK, bool REDUCE, bool ZERO, int NT>
__device__ __forceinline__ void run32(const Smem<true>& S, int pb, float k, float eps2, bool excl,
                                      const float2 (&tg)[kMaxNT][3], float2 (&acc)[NT][2]) {
#pragma unroll (ZERO ? 1 : 2)
  for (int u = 0; u < 4; u++) {
    const float4 a = S.A[pb + 4 * u], b = S.B[pb + 4 * u];
    const float2 qi = S.Q[pb + 4 * u], qr = make_float2(b.z, b.w);
    const float2 sx = make_float2(a.x, a.y), sy = make_float2(a.z, a.w), sz = make_float2(b.x, b.y);
#pragma unroll
    for (int t = 0; t < NT; t++) {
      const float2 dx = __fadd2_rn(tg[t][0], sx), dy = __fadd2_rn(tg[t][1], sy), dz = __fadd2_rn(tg[t][2], sz);
      float2 r2, ri;
      if (ZERO) {
        const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
        r2 = __fadd2_rn(d2, dup(eps2));
        ri.x = (excl && d2.x == 0.f) || r2.x == 0.f ? 0.f : rsqrt_ftz(r2.x);
        ri.y = (excl && d2.y == 0.f) || r2.y == 0.f ? 0.f : rsqrt_ftz(r2.y);
      } else {
        r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, dup(eps2))));
        ri = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
      }
      const float2 ph = __fmul2_rn(dup(k), __fmul2_rn(r2, ri));
      if (YUK) {  // real kernel e^{-k r} / r
        const float2 e = __fmul2_rn(make_float2(__expf(-ph.x), __expf(-ph.y)), ri);
        acc[t][0] = __ffma2_rn(qr, e, acc[t][0]);
        acc[t][1] = __ffma2_rn(qi, e, acc[t][1]);
      } else {
        float2 red = ph;
        if (REDUCE) {
          red.x = fmaf(-6.28318530717958647f, rintf(ph.x * 0.159154943091895336f), ph.x);
          red.y = fmaf(-6.28318530717958647f, rintf(ph.y * 0.159154943091895336f), ph.y);
        }
        float2 sn, cs;
        __sincosf(red.x, &sn.x, &cs.x);
        __sincosf(red.y, &sn.y, &cs.y);
        sn = __fmul2_rn(sn, ri);
        cs = __fmul2_rn(cs, ri);
        const float2 ns = make_float2(-sn.x, -sn.y);
        acc[t][0] = __ffma2_rn(qr, cs, __ffma2_rn(qi, ns, acc[t][0]));
        acc[t][1] = __ffma2_rn(qr, sn, __ffma2_rn(qi, cs, acc[t][1]));
      }
    }
  }
}

// 1/sqrt(a), a > 0 normal: the hardware estimate (relative error below 2^-19)
// and one third-order step, as p2p_f64.cu
__device__ __forceinline__ double inv_sqrt(double a) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  const double e = fma(-(a * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// sin and cos of x >= 0 in 30 FP64 operations (the library's general routine takes
// several times as many).  Cody and Waite's reduction by multiples of pi/2 in two
// parts (W. J. Cody, W. Waite, Software Manual for the Elementary Functions,
// 1980), then the Taylor series on [-pi/4, pi/4] up to x^17 and x^16: the next
// terms are below 2^-63 and 2^-58.  The reduced argument carries x's own
// rounding, as any reduction does.  For x <= kPhaseMax, where two parts of pi/2 do.
constexpr double kPhaseMax = 1e5;
__device__ __forceinline__ void sincos_phase(double x, double& sn, double& cs) {
  constexpr double kMagic = 6755399441055744.0;  // 1.5 * 2^52: rounds to an integer in the low word
  const double t = fma(x, M_2_PI, kMagic), n = t - kMagic;
  const int q = __double2loint(t);
  const double h = fma(-n, M_PI_2, x), lo = 6.123233995736766e-17;  // pi/2 - M_PI_2
  const double r = fma(-n, lo, h), e = fma(-n, lo, h - r), z = r * r;  // r + e: the reduced argument
  double a = fma(z, 1.0 / 355687428096000.0, -1.0 / 1307674368000.0);  // 1/17!, 1/15!
  a = fma(z, a, 1.0 / 6227020800.0);
  a = fma(z, a, -1.0 / 39916800.0);
  a = fma(z, a, 1.0 / 362880.0);
  a = fma(z, a, -1.0 / 5040.0);
  a = fma(z, a, 1.0 / 120.0);
  a = fma(z, a, -1.0 / 6.0);
  const double s = r + fma(r * z, a, e);
  double b = fma(z, 1.0 / 20922789888000.0, -1.0 / 87178291200.0);  // 1/16!, 1/14!
  b = fma(z, b, 1.0 / 479001600.0);
  b = fma(z, b, -1.0 / 3628800.0);
  b = fma(z, b, 1.0 / 40320.0);
  b = fma(z, b, -1.0 / 720.0);
  b = fma(z, b, 1.0 / 24.0);
  const double w = fma(z, -0.5, 1.0);  // 1 - z / 2, and what its rounding lost
  const double c = w + fma(z * z, b, fma(-r, e, fma(z, -0.5, 1.0 - w)));
  const double u = q & 1 ? c : s, v = q & 1 ? s : c;
  sn = q & 2 ? -u : u;
  cs = (q + 1) & 2 ? -v : v;
}

// A coordinate this close to zero can differ by less than 2^-60 from another, so that a squared distance underflows
// in FP32; other coordinates are equal or at least that far apart.
__device__ __forceinline__ bool tiny(float c) { return c != 0.f && fabsf(c) < 0x1p-36f; }
__device__ __forceinline__ bool tiny(const float4& x) { return tiny(x.x) || tiny(x.y) || tiny(x.z); }

// The lane's sources of the chunk's runs w, w + m, ... of nrun against one target, for any r^2: the library's inverse
// root takes subnormal ones.  Out of line, so that the loops above keep their registers.
template <bool YUK>
__device__ __noinline__ double2 near_zero_runs(const Smem<true>& S, int nrun, int s, int w, int m, float k, float eps2,
                                               bool excl, float x, float y, float z) {
  double2 sum = make_double2(0.0, 0.0);
#pragma unroll 1
  for (int r = w; r < nrun; r += m) {
    float re = 0.f, im = 0.f;
#pragma unroll 1
    for (int u = 0; u < 8; u++) {
      const int pb = 16 * r + s + 4 * (u >> 1), h = u & 1;
      const float4 a = S.A[pb], b = S.B[pb];
      const float2 q = S.Q[pb];
      const float dx = x + (h ? a.y : a.x), dy = y + (h ? a.w : a.z), dz = z + (h ? b.y : b.x);
      const float d2 = dx * dx + dy * dy + dz * dz, r2 = d2 + eps2;
      if ((excl && d2 == 0.f) || r2 == 0.f) continue;
      const float ri = rsqrtf(r2), ph = k * (r2 * ri), qr = h ? b.w : b.z, qi = h ? q.y : q.x;
      if (YUK) {
        const float e = __expf(-ph) * ri;
        re = fmaf(qr, e, re);
        im = fmaf(qi, e, im);
      } else {
        float sn, cs;
        __sincosf(fmaf(-6.28318530717958647f, rintf(ph * 0.159154943091895336f), ph), &sn, &cs);
        re += (qr * cs - qi * sn) * ri;
        im += (qr * sn + qi * cs) * ri;
      }
    }
    sum.x += (double)re;
    sum.y += (double)im;
  }
  return sum;
}

// the lane's 8 sources of a run of 32 (j0, j0 + 4, ...) against its NT targets
template <bool YUK, bool ZERO, int NT>
__device__ __forceinline__ void run32(const Smem<false>& S, int j0, double k, double eps2, bool excl,
                                      const double (&tg)[kMaxNT][3], double (&acc)[kMaxNT][2]) {
#pragma unroll 1
  for (int u = 0; u < 32 / kS; u++) {
    const double2 a = S.A[j0 + kS * u], b = S.B[j0 + kS * u];
    const double qi = S.Q[j0 + kS * u];
    // in steps over all targets, without branches, so that their serial chains
    // (estimate, step, reduction, series) overlap: few warps run in this form
    double ri[NT], ph[NT];
    bool on[NT], big = false;
#pragma unroll
    for (int t = 0; t < NT; t++) {
      const double dx = tg[t][0] - a.x, dy = tg[t][1] - a.y, dz = tg[t][2] - b.x;
      const double d2 = fma(dx, dx, fma(dy, dy, dz * dz)), r2 = d2 + eps2;
      ri[t] = inv_sqrt(r2);
      on[t] = true;
      if (ZERO) {  // below the estimate's range: the library's, and no term at zero
        if (r2 < 0x1p-1000) ri[t] = 1.0 / sqrt(r2);
        on[t] = !((excl && d2 == 0.0) || r2 == 0.0);
      }
      ph[t] = on[t] ? k * (r2 * ri[t]) : 0.0;
      big |= !(ph[t] <= kPhaseMax);
    }
    double sn[NT], cs[NT];
    if (YUK) {
#pragma unroll
      for (int t = 0; t < NT; t++) cs[t] = exp(-ph[t]);
    } else if (big) {
#pragma unroll
      for (int t = 0; t < NT; t++) sincos(ph[t], &sn[t], &cs[t]);
    } else {
#pragma unroll
      for (int t = 0; t < NT; t++) sincos_phase(ph[t], sn[t], cs[t]);
    }
#pragma unroll
    for (int t = 0; t < NT; t++) {
      if (ZERO && !on[t]) continue;
      cs[t] *= ri[t];
      if (YUK) {
        acc[t][0] = fma(b.y, cs[t], acc[t][0]);
        acc[t][1] = fma(qi, cs[t], acc[t][1]);
      } else {
        sn[t] *= ri[t];
        acc[t][0] = fma(b.y, cs[t], fma(-qi, sn[t], acc[t][0]));
        acc[t][1] = fma(b.y, sn[t], fma(qi, cs[t], acc[t][1]));
      }
    }
  }
}

// pad: where the list's padding lies, 16 leaf sides from the targets (the phase stays moderate), no charge.
// Returns whether any thread's near0 is set or a source has a coordinate close to zero.
__device__ __forceinline__ bool stage(Smem<true>& S, int c0, int c1, bool near0, float4 pad,
                                      const float4* __restrict__ spos, const float2* __restrict__ q) {
  __syncthreads();  // the previous chunk's readers are done
  for (int u = threadIdx.x; u < (c1 - c0) / 2; u += 32 * max_warps(true)) {
    float4 x[2];
    float2 qq[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int j = S.src.locate(c0 + 2 * u + h, c1);
      x[h] = pad;
      qq[h] = make_float2(0.f, 0.f);
      if (j >= 0) {
        x[h] = spos[j];
        qq[h] = q[j];
        near0 |= tiny(x[h]);
      }
    }
    S.A[u] = make_float4(-x[0].x, -x[1].x, -x[0].y, -x[1].y);
    S.B[u] = make_float4(-x[0].z, -x[1].z, qq[0].x, qq[1].x);
    S.Q[u] = make_float2(qq[0].y, qq[1].y);
  }
  return __syncthreads_or(near0);
}

__device__ __forceinline__ bool stage(Smem<false>& S, int c0, int c1, bool, float4 pad, const float4* __restrict__ spos,
                                      const float2* __restrict__ q) {
  __syncthreads();
  for (int u = threadIdx.x; u < c1 - c0; u += blockDim.x) {
    const int j = S.src.locate(c0 + u, c1);
    float4 x = pad;
    float2 qq = make_float2(0.f, 0.f);
    if (j >= 0) {
      x = spos[j];
      qq = q[j];
    }
    S.A[u] = make_double2(x.x, x.y);
    S.B[u] = make_double2(x.z, qq.x);
    S.Q[u] = qq.y;
  }
  __syncthreads();
  return false;  // squared differences of floats are normal in FP64
}

// The team tile's runs of the chunk [c0, c1): runs k, k + m, ..., the own
// leaf's runs (below self_end) and the list's last one (from last on) with the
// zero-distance test.
template <bool YUK, bool REDUCE, int NT>
__device__ __forceinline__ void tile_runs(const Smem<true>& S, int c0, int c1, int self_end, int last, int s, int w, int m, float k,
                                          float eps2, bool excl, const float2 (&tg)[kMaxNT][3], double (&P)[kMaxNT][2]) {
  for (int r = (c0 >> 5) + w; r < (c1 >> 5);) {  // c0 / 32 is a multiple of m
    float2 acc[NT][2];
#pragma unroll
    for (int t = 0; t < NT; t++) acc[t][0] = acc[t][1] = make_float2(0.f, 0.f);
    for (int i = 0; i < 4 && r < (c1 >> 5); i++, r += m) {  // 4 runs: 16 sources in each of a lane's two sums
      const int pb = ((r * 32 - c0) >> 1) + s;
      if (r * 32 < self_end || r * 32 >= last) run32<YUK, REDUCE, true, NT>(S, pb, k, eps2, excl, tg, acc);
      else run32<YUK, REDUCE, false, NT>(S, pb, k, eps2, excl, tg, acc);
    }
#pragma unroll
    for (int t = 0; t < NT; t++) {
      P[t][0] += (double)(acc[t][0].x + acc[t][0].y);
      P[t][1] += (double)(acc[t][1].x + acc[t][1].y);
    }
  }
}
template <bool YUK, bool REDUCE, int NT>
__device__ __forceinline__ void tile_runs(const Smem<false>& S, int c0, int c1, int self_end, int last, int s, int w, int m, double k,
                                          double eps2, bool excl, const double (&tg)[kMaxNT][3], double (&P)[kMaxNT][2]) {
  for (int r = (c0 >> 5) + w; r < (c1 >> 5); r += m) {
    if (r * 32 < self_end || r * 32 >= last) run32<YUK, true, NT>(S, r * 32 - c0 + s, k, eps2, excl, tg, P);
    else run32<YUK, false, NT>(S, r * 32 - c0 + s, k, eps2, excl, tg, P);
  }
}

template <bool F32>
struct Num;
template <>
struct Num<true> {
  using T = float;
  using V = float2;
  static __device__ __forceinline__ V make(float v) { return dup(v); }
};
template <>
struct Num<false> {
  using T = double;
  using V = double;
  static __device__ __forceinline__ V make(float v) { return (double)v; }
};

template <bool F32, bool YUK, bool REDUCE>
__global__ void __launch_bounds__(32 * max_warps(F32)) helm_p2p(float k, float eps2, int excl, float far, const int2* __restrict__ work,
                                                     const int2* __restrict__ leaf_i, const int2* __restrict__ leaf_j,
                                                     const int* __restrict__ list, const float4* __restrict__ tpos,
                                                     const float4* __restrict__ spos, const float2* __restrict__ q,
                                                     double2* __restrict__ pot) {
  using T = typename Num<F32>::T;
  __shared__ Smem<F32> S;
  const int2 wk = work[blockIdx.x];
  const int b = wk.x;
  int2 li = leaf_i[b];
  float4 pad = tpos[li.x];
  pad.x += far;
  li.x += wk.y;
  li.y = min(kItem, li.y - wk.y);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane & (kG - 1), s = lane / kG;
  if (warp == 0) S.src.build(b, list, leaf_j, lane);
  __syncthreads();
  const int self_end = S.src.self_end(), vlen = S.src.length();
  const int nchunk = (vlen + kCap - 1) / kCap;
  // teams of m warps share a tile of up to 4 groups of targets and split its runs
  const int ng = (li.y + kG - 1) / kG;
  const int NW = F32 ? 4 : blockDim.x >> 5;
  const int m = ng <= kMaxNT ? NW : ng <= 2 * kMaxNT ? NW / 2 : NW / 4;  // block-uniform
  const int nteam = NW / m, team = warp / m, w = warp % m;
  const int ga = team * ng / nteam, ntl = (team + 1) * ng / nteam - ga;  // at most 4 groups: li.y <= 128
  typename Num<F32>::V tg[kMaxNT][3];
  double P[kMaxNT][2];
  bool near0 = F32 && eps2 > 0.f && eps2 < 0x1p-126f;
#pragma unroll
  for (int t = 0; t < kMaxNT; t++) {
    const int it = (ga + t) * kG + g;
    const float4 x = t < ntl && it < li.y ? tpos[li.x + it] : make_float4(0.f, 0.f, 0.f, 0.f);
    near0 |= F32 && tiny(x);
    tg[t][0] = Num<F32>::make(x.x);
    tg[t][1] = Num<F32>::make(x.y);
    tg[t][2] = Num<F32>::make(x.z);
    P[t][0] = P[t][1] = 0.0;
  }
  for (int ch = 0; ch < nchunk; ch++) {
    const int c0 = ch * kCap, c1 = min(vlen, c0 + kCap);
    const bool sub = stage(S, c0, c1, near0, pad, spos, q);  // block-uniform
    if constexpr (F32) {
      if (sub) {
#pragma unroll
        for (int t = 0; t < kMaxNT; t++) {
          if (t >= ntl) break;
          const double2 v = near_zero_runs<YUK>(S, (c1 - c0) >> 5, s, w, m, k, eps2, excl, tg[t][0].x, tg[t][1].x,
                                                tg[t][2].x);
          P[t][0] += v.x;
          P[t][1] += v.y;
        }
        continue;
      }
    }
    switch (ntl) {
      case 0: break;
      case 1: tile_runs<YUK, REDUCE, 1>(S, c0, c1, self_end, vlen - 32, s, w, m, (T)k, (T)eps2, excl, tg, P); break;
      case 2: tile_runs<YUK, REDUCE, 2>(S, c0, c1, self_end, vlen - 32, s, w, m, (T)k, (T)eps2, excl, tg, P); break;
      case 3: tile_runs<YUK, REDUCE, 3>(S, c0, c1, self_end, vlen - 32, s, w, m, (T)k, (T)eps2, excl, tg, P); break;
      default: tile_runs<YUK, REDUCE, 4>(S, c0, c1, self_end, vlen - 32, s, w, m, (T)k, (T)eps2, excl, tg, P); break;
    }
  }
  // add the 4 streams' sums of each target, then the team's warps through shared memory
#pragma unroll
  for (int t = 0; t < kMaxNT; t++)
#pragma unroll
    for (int c = 0; c < 2; c++) {
      P[t][c] += __shfl_xor_sync(0xffffffffu, P[t][c], 8);
      P[t][c] += __shfl_xor_sync(0xffffffffu, P[t][c], 16);
    }
  if (m > 1) {  // block-uniform
    if (s == 0 && w > 0) {
#pragma unroll
      for (int t = 0; t < kMaxNT; t++)
#pragma unroll
        for (int c = 0; c < 2; c++) S.red[warp - 1][t][c][g] = P[t][c];
    }
    __syncthreads();
    if (w == 0 && s == 0) {
      for (int v = 1; v < m; v++)
#pragma unroll
        for (int t = 0; t < kMaxNT; t++)
#pragma unroll
          for (int c = 0; c < 2; c++) P[t][c] += S.red[warp + v - 1][t][c][g];
    }
  }
  if (w == 0 && s == 0) {
    const double coef = 0.25 / M_PI;
#pragma unroll
    for (int t = 0; t < kMaxNT; t++) {
      const int it = (ga + t) * kG + g;
      if (t < ntl && it < li.y) pot[li.x + it] = make_double2(coef * P[t][0], coef * P[t][1]);
    }
  }
}

}  // namespace

void launch_helm_p2p(bool f32, bool yuk, float k, float eps2, bool excl, float leaf_side, int nwork,
                     const int2* work, const int2* leaf_i, const int2* leaf_j, const int* list, const float4* tpos,
                     const float4* spos, const float* qs, double* pot, cudaStream_t st) {
  if (nwork <= 0) return;
  // points of neighbouring leaves lie at most 2 sqrt(3) leaf sides apart: below pi / k (with a margin for the float
  // phase) the reduction is the identity and is left out
  const double rmax = std::sqrt(12.0 * (double)leaf_side * leaf_side + (double)eps2);
  const bool reduce = !((double)k * rmax < 0.999 * M_PI);
  auto go = [&](auto kern) {
    kern<<<nwork, !f32 && nwork <= kFewItems ? 256 : 128, 0, st>>>(k, eps2, excl ? 1 : 0, 16.f * leaf_side, work, leaf_i, leaf_j, list, tpos, spos, (const float2*)qs,
                                     (double2*)pot);
  };
  if (f32 && !yuk && reduce) go(helm_p2p<true, false, true>);
  else if (f32 && !yuk) go(helm_p2p<true, false, false>);
  else if (f32) go(helm_p2p<true, true, false>);
  else if (!yuk) go(helm_p2p<false, false, false>);
  else go(helm_p2p<false, true, false>);
  FMMB_CHECK_LAUNCH();
}

}  // namespace fmmb
