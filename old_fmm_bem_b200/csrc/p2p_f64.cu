// Near-field P2P in FP64 (the plain-FP64 form of every Laplace kernel).
//
// The sums of the reference's P2P kernels (kernel/G_p2p.cxx:12-37,
// kernel/Gni_p2p.cxx:12-28, kernel/Gnj_p2p.cxx:12-28) over the 27-slot
// neighbour lists, everything after the coordinate difference in FP64.  In
// reference semantics the difference itself is taken in FP32, as the
// reference does (kernel/G_p2p.cxx:21-23).
//
// Bound: the FP64 pipe (64 FMA lanes per clock and SM).  A pair of G with its
// gradient needs 18 FP64 operations -- 3 differences, 3 for r^2, 5 for the
// inverse root, 1 for q/r, 2 for q/r^3, 4 sums -- so everything else is kept off
// that pipe: sources are converted to FP64 once, when they are staged (in
// accurate semantics), the charges are staged times the 1/(4 pi), and 1/r is the
// hardware's 20-bit estimate with one third-order step instead of a square root
// and a division.
//
// Layout (as the mixed form's, p2p_mixed.cu): a block of 4 warps per work item
// of up to 128 targets of a leaf; the sources of the neighbour leaves staged as
// one list in chunks; a warp is 8 target lanes x 4 source streams, each lane
// holding NT <= 4 targets, so one shared-memory read of a source serves NT pairs
// and a leaf of 24 or 64 targets still fills the lanes (one thread per target
// left 104 or 64 of a block's 128 threads idle); the warps form teams that share
// a tile of targets and split its runs of sources.
//
// Measured against one thread per target with a square root and a division per
// pair (one B200, whole FP64 evaluate with gradient): 262,144 clustered points at
// p = 12, depth 5 (1.54 G pairs) 13.15 -> 8.87 ms; 32,768 uniform points at p = 8,
// depth 3 (43.5 M pairs) 1.08 -> 0.59 ms.  The test for r = 0 and subnormal r^2
// only where a pair can coincide, the targets' own leaf: this kernel with the
// present far field beside it, 2.84 -> 2.62 and 0.281 -> 0.257 ms.
#include <cuda_runtime.h>

#include "internal.h"
#include "kernels.h"
#include "p2p_list.cuh"

namespace fmmb {
namespace {

constexpr int kItem = 128;   // targets of a work item
constexpr int kMaxWarps = 8;
// Warps of a block: 4; 8 where all items are resident at once with 4 (4 blocks fit an
// SM by their registers) and leave the FP64 pipe short of warps.  Whole evaluate
// with 4 / 8, us: G with gradient, p = 8, 64 points a leaf: 64 items 77 / 63, 343 129 /
// 124, 512 161 / 166, 729 213 / 221; 128 a leaf: 64 items 169 / 123, 343 311 / 235, 512
// 377 / 334, 729 455 / 466; Gnj, p = 10, 64 a leaf: 216 items 204 / 105, 512 235 / 194,
// 729 258 / 258; 24 a leaf within 4 % throughout.  4,219 items (262,144 clustered
// points) 2.43 / 2.52 ms.
constexpr int kFewItems = 4 * 148;
constexpr int kG = 8;        // targets of a group (lanes g = lane % 8)
constexpr int kS = 32 / kG;  // source streams of a warp (s = lane / 8)
constexpr int kMaxNT = 4;    // groups of a tile
constexpr int kCap = 512;    // staged sources per chunk (multiple of 32 * 4)

// 1/sqrt(a) for normal a > 0: the hardware's estimate y (relative error below
// 2^-19) and the first three terms of (1 - e)^(-1/2) = 1 + e/2 + 3 e^2/8 + ...,
// e = 1 - a y^2: what is left out, 5 e^3 / 16, is below 2^-54.  (Squared
// differences of floats, at least 2^-298, are normal.)
__device__ __forceinline__ double inv_sqrt(double a) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  const double e = fma(-(a * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}
// a >= 0 of a pair that may coincide: subnormal a (a tiny softening), which the
// estimate flushes, is scaled by 2^200 first; a = 0 gives infinity
__device__ __forceinline__ double inv_sqrt_any(double a) {
  if (__double2hiint(a) >= 0x00100000) return inv_sqrt(a);
  return a > 0.0 ? inv_sqrt(a * 0x1p200) * 0x1p100 : __longlong_as_double(0x7ff0000000000000ll);
}

template <int KER, bool REF>
struct Smem {
  // accurate: (x, y), (z, c q) in FP64; reference: (x, y, z) in FP32 and c q in FP64 (c = 1/(4 pi))
  double2 A[REF ? 1 : kCap], B[REF ? 1 : kCap];
  float4 X[REF ? kCap : 1];
  double Q[REF ? kCap : 1];
  double2 N[KER == FMMB_LAPLACE_GNJ ? kCap : 1];  // source normal (x, y), z
  double NZ[KER == FMMB_LAPLACE_GNJ ? kCap : 1];
  double red[kMaxWarps - 1][kMaxNT][4][kG];  // team partial sums
  SrcList src;
};

template <bool REF>
struct Tgt {
  double x, y, z;
};
template <>
struct Tgt<true> {
  float x, y, z;
};

// One run of 32 sources: the lane's 8 sources (j0 + s, + 4, ...) against its NT targets.
// OWN: a run of the targets' own leaf, where a pair may coincide (in reference
// semantics its softening keeps r away from 0).
template <int KER, bool GRAD, bool REF, bool EXCL, bool OWN, int NT>
__device__ __forceinline__ void run32(const Smem<KER, REF>& S, int j0, double eps2, const Tgt<REF> (&tg)[kMaxNT],
                                      const double (&tn)[kMaxNT][3], double (&P)[kMaxNT][4]) {
#pragma unroll 2
  for (int u = 0; u < 32 / kS; u++) {
    const int j = j0 + kS * u;
    double sx, sy, sz, q;
    float fx, fy, fz;
    if (REF) {
      const float4 v = S.X[j];
      fx = v.x, fy = v.y, fz = v.z;
      q = S.Q[j];
    } else {
      const double2 a = S.A[j], b = S.B[j];
      sx = a.x, sy = a.y, sz = b.x, q = b.y;
    }
    double nx = 0, ny = 0, nz = 0;
    if (KER == FMMB_LAPLACE_GNJ) {
      const double2 n = S.N[j];
      nx = n.x, ny = n.y, nz = S.NZ[j];
    }
#pragma unroll
    for (int t = 0; t < NT; t++) {
      double dx, dy, dz;
      if (REF) {
        dx = (double)__fsub_rn((float)tg[t].x, fx);
        dy = (double)__fsub_rn((float)tg[t].y, fy);
        dz = (double)__fsub_rn((float)tg[t].z, fz);
      } else {
        dx = tg[t].x - sx;
        dy = tg[t].y - sy;
        dz = tg[t].z - sz;
      }
      const double r2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)));
      const double rinv = OWN && !REF ? inv_sqrt_any(r2) : inv_sqrt(r2);
      double qr = q * rinv;
      if (OWN && EXCL) {
        if (dx == 0.0 && dy == 0.0 && dz == 0.0) continue;
      }
      if (KER == FMMB_LAPLACE_G) {
        P[t][0] += qr;
        if (GRAD) {
          const double qr3 = qr * rinv * rinv;
          P[t][1] = fma(-dx, qr3, P[t][1]);
          P[t][2] = fma(-dy, qr3, P[t][2]);
          P[t][3] = fma(-dz, qr3, P[t][3]);
        }
      } else {
        // n = the target's normal (Gni) or the source's (Gnj).  Gradient w.r.t. the target
        // position: d/dx_i of q (d.n) / r^3 = q n / r^3 - 3 q (d.n) d / r^5
        if (KER == FMMB_LAPLACE_GNI) nx = tn[t][0], ny = tn[t][1], nz = tn[t][2];
        const double dot = fma(dx, nx, fma(dy, ny, dz * nz));
        const double rinv2 = rinv * rinv, qr3 = qr * rinv2;
        P[t][0] = fma(dot, qr3, P[t][0]);
        if (GRAD) {
          const double c = -3.0 * dot * qr3 * rinv2;
          P[t][1] = fma(qr3, nx, fma(c, dx, P[t][1]));
          P[t][2] = fma(qr3, ny, fma(c, dy, P[t][2]));
          P[t][3] = fma(qr3, nz, fma(c, dz, P[t][3]));
        }
      }
    }
  }
}

template <int KER, bool REF>
__device__ void stage(Smem<KER, REF>& S, int c0, int c1, const float4* __restrict__ spos,
                      const float4* __restrict__ snrm, const float* __restrict__ qs, double coef) {
  __syncthreads();  // the previous chunk's readers are done
  for (int u = threadIdx.x; u < c1 - c0; u += blockDim.x) {
    const int j = S.src.locate(c0 + u, c1);
    float4 x = make_float4(1e18f, 0.f, 0.f, 0.f), n = make_float4(0.f, 0.f, 0.f, 0.f);  // padding: no charge
    float q = 0.f;
    if (j >= 0) {
      x = spos[j];
      q = qs[j];
      if (KER == FMMB_LAPLACE_GNJ) n = snrm[j];
    }
    const double cq = coef * (double)q;
    if (REF) {
      S.X[u] = x;
      S.Q[u] = cq;
    } else {
      S.A[u] = make_double2(j >= 0 ? (double)x.x : 1e100, x.y);  // padding: farther off than any float
      S.B[u] = make_double2(x.z, cq);
    }
    if (KER == FMMB_LAPLACE_GNJ) {
      S.N[u] = make_double2(n.x, n.y);
      S.NZ[u] = n.z;
    }
  }
  __syncthreads();
}

// The team tile's runs of the chunk [c0, c1): runs k, k + m, ..., the own
// leaf's runs (below self_end) with the coincident-point test.
template <int KER, bool GRAD, bool REF, bool EXCL, int NT>
__device__ __forceinline__ void tile_runs(const Smem<KER, REF>& S, int c0, int c1, int self_end, int s, int k, int m,
                                          double eps2, const Tgt<REF> (&tg)[kMaxNT], const double (&tn)[kMaxNT][3],
                                          double (&P)[kMaxNT][4]) {
  for (int r = (c0 >> 5) + k; r < (c1 >> 5); r += m) {  // c0 / 32 is a multiple of m
    const int j0 = r * 32 - c0 + s;
    if (r * 32 < self_end)
      run32<KER, GRAD, REF, EXCL, true, NT>(S, j0, eps2, tg, tn, P);
    else
      run32<KER, GRAD, REF, EXCL, false, NT>(S, j0, eps2, tg, tn, P);
  }
}

template <int KER, bool GRAD, bool REF, bool EXCL>
__global__ void __launch_bounds__(32 * kMaxWarps) p2p_f64(const int2* __restrict__ work, const int2* __restrict__ leaf_i,
                                                    const int2* __restrict__ leaf_j, const int* __restrict__ list,
                                                    const float4* __restrict__ tpos, const float4* __restrict__ tnrm,
                                                    const float4* __restrict__ spos, const float4* __restrict__ snrm,
                                                    const float* __restrict__ qs, double eps2, double coef,
                                                    double* __restrict__ pot, double* __restrict__ grad, int ni) {
  constexpr int NC = GRAD ? 4 : 1;
  __shared__ Smem<KER, REF> S;
  const int2 wk = work[blockIdx.x];
  const int b = wk.x;
  int2 li = leaf_i[b];
  li.x += wk.y;
  li.y = min(kItem, li.y - wk.y);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane & (kG - 1), s = lane / kG;
  if (warp == 0) S.src.build(b, list, leaf_j, lane);
  __syncthreads();
  const int self_end = S.src.self_end(), vlen = S.src.length();
  const int nchunk = (vlen + kCap - 1) / kCap;
  // teams of m warps share a tile of up to 4 groups of targets and split its runs
  const int ng = (li.y + kG - 1) / kG;
  const int nw = blockDim.x >> 5;  // 4 or 8
  const int m = ng <= kMaxNT ? nw : ng <= 2 * kMaxNT ? nw / 2 : nw / 4;  // block-uniform
  const int nteam = nw / m, team = warp / m, k = warp % m;
  const int ga = team * ng / nteam, ntl = (team + 1) * ng / nteam - ga;  // at most 4 groups: li.y <= 128
  Tgt<REF> tg[kMaxNT];
  double tn[kMaxNT][3], P[kMaxNT][4];
#pragma unroll
  for (int t = 0; t < kMaxNT; t++) {
    const int it = (ga + t) * kG + g;
    const bool on = t < ntl && it < li.y;
    const float4 x = on ? tpos[li.x + it] : make_float4(0.f, 0.f, 0.f, 0.f);
    tg[t].x = x.x;
    tg[t].y = x.y;
    tg[t].z = x.z;
    if (KER == FMMB_LAPLACE_GNI) {
      const float4 n = on ? tnrm[li.x + it] : make_float4(0.f, 0.f, 0.f, 0.f);
      tn[t][0] = n.x;
      tn[t][1] = n.y;
      tn[t][2] = n.z;
    }
#pragma unroll
    for (int c = 0; c < 4; c++) P[t][c] = 0.0;
  }
  for (int ch = 0; ch < nchunk; ch++) {
    const int c0 = ch * kCap, c1 = min(vlen, c0 + kCap);
    stage<KER, REF>(S, c0, c1, spos, snrm, qs, coef);
    switch (ntl) {
      case 0: break;
      case 1: tile_runs<KER, GRAD, REF, EXCL, 1>(S, c0, c1, self_end, s, k, m, eps2, tg, tn, P); break;
      case 2: tile_runs<KER, GRAD, REF, EXCL, 2>(S, c0, c1, self_end, s, k, m, eps2, tg, tn, P); break;
      case 3: tile_runs<KER, GRAD, REF, EXCL, 3>(S, c0, c1, self_end, s, k, m, eps2, tg, tn, P); break;
      default: tile_runs<KER, GRAD, REF, EXCL, 4>(S, c0, c1, self_end, s, k, m, eps2, tg, tn, P); break;
    }
  }
  // add the 4 streams' sums of each target, then the team's warps through shared memory
#pragma unroll
  for (int t = 0; t < kMaxNT; t++)
#pragma unroll
    for (int c = 0; c < NC; c++) {
      P[t][c] += __shfl_xor_sync(0xffffffffu, P[t][c], 8);
      P[t][c] += __shfl_xor_sync(0xffffffffu, P[t][c], 16);
    }
  if (m > 1) {  // block-uniform
    if (s == 0 && k > 0) {
#pragma unroll
      for (int t = 0; t < kMaxNT; t++)
#pragma unroll
        for (int c = 0; c < NC; c++) S.red[warp - 1][t][c][g] = P[t][c];
    }
    __syncthreads();
    if (k == 0 && s == 0) {
      for (int w = 1; w < m; w++)
#pragma unroll
        for (int t = 0; t < kMaxNT; t++)
#pragma unroll
          for (int c = 0; c < NC; c++) P[t][c] += S.red[warp + w - 1][t][c][g];
    }
  }
  if (k == 0 && s == 0) {
#pragma unroll
    for (int t = 0; t < kMaxNT; t++) {
      const int it = (ga + t) * kG + g;
      if (t < ntl && it < li.y) {
        const int i = li.x + it;
        pot[i] = P[t][0];
        if (GRAD) {
          grad[i] = P[t][1];
          grad[ni + (size_t)i] = P[t][2];
          grad[2 * (size_t)ni + i] = P[t][3];
        }
      }
    }
  }
}

}  // namespace

void launch_p2p_f64(int kernel, int nwork, const int2* work, const int2* leaf_i, const int2* leaf_j, const int* list,
                    const float4* tpos, const float4* tnrm, const float4* spos, const float4* snrm, const float* qs,
                    const Sem& s, double* pot, double* grad, int ni, cudaStream_t st) {
  if (nwork <= 0) return;
  auto go = [&](auto k) {
    k<<<nwork, nwork <= kFewItems ? 256 : 128, 0, st>>>(work, leaf_i, leaf_j, list, tpos, tnrm, spos, snrm, qs, s.eps2, s.coef, pot, grad,
                                  ni);
  };
  auto pick = [&](auto ker) {  // reference semantics: self pairs included
    constexpr int K = decltype(ker)::value;
    if (s.ref) {
      if (grad) go(p2p_f64<K, true, true, false>);
      else go(p2p_f64<K, false, true, false>);
    } else if (s.excl_self) {
      if (grad) go(p2p_f64<K, true, false, true>);
      else go(p2p_f64<K, false, false, true>);
    } else {
      if (grad) go(p2p_f64<K, true, false, false>);
      else go(p2p_f64<K, false, false, false>);
    }
  };
  if (kernel == FMMB_LAPLACE_G) pick(std::integral_constant<int, FMMB_LAPLACE_G>{});
  else if (kernel == FMMB_LAPLACE_GNI) pick(std::integral_constant<int, FMMB_LAPLACE_GNI>{});
  else pick(std::integral_constant<int, FMMB_LAPLACE_GNJ>{});
  FMMB_CHECK_LAUNCH();
}

}  // namespace fmmb
