// Near field for many right-hand sides at once (mixed form, Laplace kernels).
//
// The same sums as p2p_mixed.cu (kernel/G_p2p.cxx:12-37, Gni_p2p.cxx:12-28,
// Gnj_p2p.cxx:12-28) for R charge vectors in one pass: the pair geometry --
// distance, inverse distance, the kernel's factors -- is computed once per pair
// and applied to the R charges of the source, so a GMRES block of R iterates
// costs little more than one.
//
// Layout (as p2p_mixed.cu's): one block of 8 warps per work item of up to 128
// targets of a leaf; the neighbour leaves' sources staged as one list
// (p2p_list.cuh) in chunks, packed in pairs with their R charges; a warp is 8
// target lanes x 4 source streams, a lane holding 2 targets, so that one
// shared-memory read of a pair of sources and its charges serves 4 pairs of
// points; the two-lane FP32 instructions take the two sources.  Teams of warps
// share a tile of 16 targets where a leaf has fewer than 65.  A lane's two sums
// are added in FP32 and promoted to FP64 after at most 8 runs (32 sources in each),
// 4 where a leaf has 33 to 64 targets, so that a FP32 chain is no longer than such a
// leaf; the components of the 4 streams are added in FP64 and dealt to the streams'
// lanes.  Zero-distance pairs, which only the own leaf's runs can hold, are skipped
// (their inverse distance is taken as 0) when the plan excludes them.
//
// Rounding error of the potential of 8, 33, 64, 100 positive charges a leaf: 0.9, 1.1,
// 0.9, 1.2 e-8 (one target per thread, chains of one leaf and at most 128 sources: 1.2,
// 1.9, 2.5, 3.1; 16 runs, the streams added in FP32: 1.6, 2.5, 1.8, 2.5, for 1 to 2 %
// less time).
//
// Bound: the FP32 pipe: 12 + R lane operations a pair for the normal-derivative
// kernels, 13 + 4 R for G with its gradient.  Measured against one target per
// thread, two block barriers per neighbour leaf and scalar pair arithmetic: Gni,
// 8 right-hand sides, 428,400 points on 16 surfaces (1.28 G pairs), this kernel
// alone on one B200: 1.58 -> 1.39 ms.
#include <cuda_runtime.h>

#include "internal.h"
#include "kernels.h"
#include "p2p_list.cuh"

namespace fmmb {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kG = 8;        // targets of a group (lanes g = lane % 8)
constexpr int kNT = 2;       // groups of a tile
constexpr int kTargets = 128;  // of a work item: 8 tiles of 16
constexpr int kCap = 512;    // staged sources per chunk (multiple of 32 * 8)

__device__ __forceinline__ float rsqrt_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float2 dup(float v) { return make_float2(v, v); }

// Sources j, j + 1 (even j): (-x_j, -x_j+1, -y_j, -y_j+1), (-z_j, -z_j+1), the
// charges (q_j, q_j+1) of each right-hand side, the normals for Gnj.
template <int KER, int R>
struct Smem {
  static constexpr int NP = kCap / 2;
  static constexpr bool NRM = KER == FMMB_LAPLACE_GNJ;
  float4 A[NP];
  float2 Z[NP];
  float2 Q[R][NP];
  float4 M[NRM ? NP : 1];   // (nx_j, nx_j+1, ny_j, ny_j+1)
  float2 MZ[NRM ? NP : 1];
  SrcList src;
};

struct Tgt {
  float2 x, y, z, nx, ny, nz;  // coordinates and (Gni) normal, in both lanes
};

template <int KER, int R, int NC, bool EXCL>
__device__ __forceinline__ void run32(const Smem<KER, R>& S, int pb, const Tgt (&tg)[kNT], float2 e2,
                                      float2 (&acc)[kNT][R][NC]) {
#pragma unroll 1
  for (int u = 0; u < 4; u++) {
    const int pi = pb + 4 * u;
    const float4 a = S.A[pi];
    const float2 sx = make_float2(a.x, a.y), sy = make_float2(a.z, a.w), sz = S.Z[pi];
    float2 q[R];
#pragma unroll
    for (int r = 0; r < R; r++) q[r] = S.Q[r][pi];
    float2 mx, my, mz;
    if (KER == FMMB_LAPLACE_GNJ) {
      const float4 m = S.M[pi];
      mx = make_float2(m.x, m.y);
      my = make_float2(m.z, m.w);
      mz = S.MZ[pi];
    }
#pragma unroll
    for (int t = 0; t < kNT; t++) {
      const float2 dx = __fadd2_rn(tg[t].x, sx), dy = __fadd2_rn(tg[t].y, sy), dz = __fadd2_rn(tg[t].z, sz);
      const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, EXCL ? __fmul2_rn(dz, dz) : __ffma2_rn(dz, dz, e2)));
      const float2 r2 = EXCL ? __fadd2_rn(d2, e2) : d2;
      float2 ri = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
      if (EXCL && fminf(d2.x, d2.y) == 0.f) {  // the same point, or a square that underflows
        if (d2.x == 0.f && !(r2.x > 0.f && apart(dx.x, dy.x, dz.x))) ri.x = 0.f;
        if (d2.y == 0.f && !(r2.y > 0.f && apart(dx.y, dy.y, dz.y))) ri.y = 0.f;
      }
      float2 kv[NC];
      if (KER == FMMB_LAPLACE_G) {
        kv[0] = ri;
        if (NC == 4) {
          const float2 r3 = __fmul2_rn(__fmul2_rn(ri, ri), ri);
          kv[NC == 4 ? 1 : 0] = __fmul2_rn(dx, r3);
          kv[NC == 4 ? 2 : 0] = __fmul2_rn(dy, r3);
          kv[NC == 4 ? 3 : 0] = __fmul2_rn(dz, r3);
        }
      } else {
        if (KER == FMMB_LAPLACE_GNI) mx = tg[t].nx, my = tg[t].ny, mz = tg[t].nz;
        const float2 dot = __ffma2_rn(dx, mx, __ffma2_rn(dy, my, __fmul2_rn(dz, mz)));
        kv[0] = __fmul2_rn(dot, __fmul2_rn(__fmul2_rn(ri, ri), ri));
      }
#pragma unroll
      for (int r = 0; r < R; r++)
#pragma unroll
        for (int c = 0; c < NC; c++) acc[t][r][c] = __ffma2_rn(q[r], kv[c], acc[t][r][c]);
    }
  }
}

template <int KER, int R>
__device__ void stage(Smem<KER, R>& S, int c0, int c1, const float4* __restrict__ spos, const float4* __restrict__ snrm,
                      const float* __restrict__ qs, int nj) {
  __syncthreads();  // the previous chunk's readers are done
  for (int u = threadIdx.x; u < (c1 - c0) / 2; u += kThreads) {
    const int j0 = S.src.locate(c0 + 2 * u, c1), j1 = S.src.locate(c0 + 2 * u + 1, c1);
    const float4 far = make_float4(1e18f, 1e18f, 1e18f, 0.f);  // padding: far, no charge
    const float4 x0 = j0 >= 0 ? spos[j0] : far, x1 = j1 >= 0 ? spos[j1] : far;
    S.A[u] = make_float4(-x0.x, -x1.x, -x0.y, -x1.y);
    S.Z[u] = make_float2(-x0.z, -x1.z);
#pragma unroll
    for (int r = 0; r < R; r++)
      S.Q[r][u] = make_float2(j0 >= 0 ? qs[(size_t)r * nj + j0] : 0.f, j1 >= 0 ? qs[(size_t)r * nj + j1] : 0.f);
    if (KER == FMMB_LAPLACE_GNJ) {
      const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 n0 = j0 >= 0 ? snrm[j0] : z4, n1 = j1 >= 0 ? snrm[j1] : z4;
      S.M[u] = make_float4(n0.x, n1.x, n0.y, n1.y);
      S.MZ[u] = make_float2(n0.z, n1.z);
    }
  }
  __syncthreads();
}

// NC: 4 for G with its gradient, else 1
template <int KER, int R, int NC, bool EXCL>
__global__ void __launch_bounds__(kThreads) p2p_multi(const int2* __restrict__ work, const int2* __restrict__ leaf_i,
                                                      const int2* __restrict__ leaf_j, const int* __restrict__ list,
                                                      const float4* __restrict__ tpos, const float4* __restrict__ tnrm,
                                                      const float4* __restrict__ spos, const float4* __restrict__ snrm,
                                                      const float* __restrict__ qs, int nj, float eps2, double coef,
                                                      double* __restrict__ pot, double* __restrict__ grad, int ni) {
  constexpr int NK = kNT * R * NC, NPL = (NK + 3) / 4;  // components of a tile's target pair; of them per stream lane
  __shared__ Smem<KER, R> S;
  __shared__ double red[kWarps][NPL][32];
  const int2 wk = work[blockIdx.x];
  const int b = wk.x;
  int2 li = leaf_i[b];
  li.x += wk.y;
  li.y = min(kTargets, li.y - wk.y);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane & (kG - 1), s = lane / kG;
  if (warp == 0) S.src.build(b, list, leaf_j, lane);
  __syncthreads();
  const int self_end = S.src.self_end(), vlen = S.src.length();
  // teams of m warps share a tile of 2 groups of targets and split its runs
  const int ng = (li.y + kG - 1) / kG;
  const int m = ng <= kNT ? 8 : ng <= 2 * kNT ? 4 : ng <= 4 * kNT ? 2 : 1;  // block-uniform
  const int nteam = kWarps / m, team = warp / m, k = warp % m;
  const int ga = team * ng / nteam, ntl = (team + 1) * ng / nteam - ga;  // at most 2 groups: li.y <= 128
  Tgt tg[kNT];
#pragma unroll
  for (int t = 0; t < kNT; t++) {
    const int it = (ga + t) * kG + g;
    const bool on = t < ntl && it < li.y;
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 x = on ? tpos[li.x + it] : z4, n = KER == FMMB_LAPLACE_GNI && on ? tnrm[li.x + it] : z4;
    tg[t] = Tgt{dup(x.x), dup(x.y), dup(x.z), dup(n.x), dup(n.y), dup(n.z)};
  }
  double P[NPL];  // components 4 i + s of the lane's two targets
#pragma unroll
  for (int i = 0; i < NPL; i++) P[i] = 0.0;
  const float2 e2 = dup(eps2);
  const int nrun = m == 2 ? 4 : 8;  // runs between promotions (with m = 4 and 8 a chunk has 4 and 2)
  for (int c0 = 0; c0 < vlen; c0 += kCap) {
    const int c1 = min(vlen, c0 + kCap);
    stage<KER, R>(S, c0, c1, spos, snrm, qs, nj);
    if (ntl == 0) continue;
    const int rend = c1 >> 5;
    for (int r = (c0 >> 5) + k; r < rend;) {  // c0 / 32 is a multiple of m
      float2 acc[kNT][R][NC];
#pragma unroll
      for (int t = 0; t < kNT; t++)
#pragma unroll
        for (int q = 0; q < R; q++)
#pragma unroll
          for (int c = 0; c < NC; c++) acc[t][q][c] = make_float2(0.f, 0.f);
      for (int i = 0; i < nrun && r < rend; i++, r += m) {
        const int pb = ((r * 32 - c0) >> 1) + s;
        if (EXCL && r * 32 < self_end) run32<KER, R, NC, true>(S, pb, tg, e2, acc);
        else run32<KER, R, NC, false>(S, pb, tg, e2, acc);
      }
      // component kk to stream kk & 3: first across streams s, s ^ 2, then s, s ^ 1
      double half[NPL][2];
#pragma unroll
      for (int i = 0; i < NPL; i++)
#pragma unroll
        for (int b = 0; b < 2; b++) {
          float v[2];
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int kk = 4 * i + 2 * h + b;
            if (kk < NK) {
              const float2 a = acc[kk / (R * NC)][(kk / NC) % R][kk % NC];
              v[h] = a.x + a.y;
            } else {
              v[h] = 0.f;
            }
          }
          const float other = __shfl_xor_sync(0xffffffffu, s & 2 ? v[0] : v[1], 16);
          half[i][b] = (double)(s & 2 ? v[1] : v[0]) + (double)other;
        }
#pragma unroll
      for (int i = 0; i < NPL; i++)
        P[i] += (s & 1 ? half[i][1] : half[i][0]) + __shfl_xor_sync(0xffffffffu, s & 1 ? half[i][0] : half[i][1], 8);
    }
  }
  if (m > 1) {  // block-uniform: the team's warps through shared memory
    if (k > 0) {
#pragma unroll
      for (int i = 0; i < NPL; i++) red[warp][i][lane] = P[i];
    }
    __syncthreads();
    if (k == 0)
      for (int w = 1; w < m; w++)
#pragma unroll
        for (int i = 0; i < NPL; i++) P[i] += red[warp + w][i][lane];
  }
  if (k != 0) return;
#pragma unroll
  for (int kk = 0; kk < NK; kk++) {
    const int t = kk / (R * NC), r = (kk / NC) % R, c = kk % NC, it = (ga + t) * kG + g;
    if ((kk & 3) != s || t >= ntl || it >= li.y) continue;
    const int i = li.x + it;
    if (c == 0) pot[(size_t)r * ni + i] = coef * P[kk / 4];
    else grad[((size_t)3 * r + c - 1) * ni + i] = -coef * P[kk / 4];  // grad(1/r) = -d / r^3
  }
}

}  // namespace

int launch_p2p_multi(int kernel, int nrhs, int nwork, const int2* work, const int2* leaf_i, const int2* leaf_j,
                     const int* list, const float4* tpos, const float4* tnrm, const float4* spos, const float4* snrm,
                     const float* qs, int nj, const Sem& s, double* pot, double* grad, int ni, cudaStream_t st) {
  if (nwork <= 0 || nrhs <= 0) return 0;
  const bool excl = s.excl_self != 0, four = kernel == FMMB_LAPLACE_G && grad;
  int launches = 0;
  // right-hand sides in groups of 8 (4 with the gradient, whose sums take four times the registers), 4, 2, 1
  for (int r0 = 0, n; r0 < nrhs; r0 += n) {
    const int left = nrhs - r0;
    n = left >= 8 && !four ? 8 : left >= 4 ? 4 : left >= 2 ? 2 : 1;
    auto go = [&](auto kern) {
      kern<<<nwork, kThreads, 0, st>>>(work, leaf_i, leaf_j, list, tpos, tnrm, spos, snrm, qs + (size_t)r0 * nj, nj,
                                       (float)s.eps2, s.coef, pot + (size_t)r0 * ni,
                                       four ? grad + (size_t)r0 * 3 * ni : nullptr, ni);
    };
    auto pick = [&](auto ker, auto nc) {
      constexpr int K = decltype(ker)::value, C = decltype(nc)::value;
      auto rhs = [&](auto e) {
        constexpr bool X = decltype(e)::value;
        if constexpr (C == 1) {
          if (n == 8) return go(p2p_multi<K, 8, C, X>);
        }
        if (n == 4) go(p2p_multi<K, 4, C, X>);
        else if (n == 2) go(p2p_multi<K, 2, C, X>);
        else go(p2p_multi<K, 1, C, X>);
      };
      if (excl) rhs(std::true_type{});
      else rhs(std::false_type{});
    };
    using One = std::integral_constant<int, 1>;
    if (four) pick(std::integral_constant<int, FMMB_LAPLACE_G>{}, std::integral_constant<int, 4>{});
    else if (kernel == FMMB_LAPLACE_G) pick(std::integral_constant<int, FMMB_LAPLACE_G>{}, One{});
    else if (kernel == FMMB_LAPLACE_GNI) pick(std::integral_constant<int, FMMB_LAPLACE_GNI>{}, One{});
    else pick(std::integral_constant<int, FMMB_LAPLACE_GNJ>{}, One{});
    FMMB_CHECK_LAUNCH();
    launches++;
  }
  return launches;
}

}  // namespace fmmb
