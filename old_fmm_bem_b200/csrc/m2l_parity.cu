// M2L in FP64: the plain-FP64 form of the Laplace kernels (and the mixed form
// above p = 15), and both forms of the Helmholtz family.
//
// The translation of a box pair at relative position D is R(-phi) T R(phi):
// R(phi) multiplies the order-m coefficients by e^{i m phi}, phi the azimuth of
// D, and T is the translation along (rho, 0, dz) -- the same for every D of one
// (rho, dz), 61 of them for the 316 relative positions (operators.cpp composes
// the reference's rotate / translate / rotate-back steps of
// kernel/m2l.cxx:30-83 for them; helmholtz.cu projects them).  T commutes with
// the reflection y -> -y, so it does not mix the even combinations of the
// orders m, -m with the odd ones:
//   Laplace (real fields): even = Re, odd = Im of E_n^m;
//   Helmholtz: even = E_n^m + E_n^-m, odd = E_n^m - E_n^-m.
// So the K x K operator becomes two blocks, (p+1)(p+2)/2 and p(p+1)/2 square:
// half the multiplications, and a fifth of the operators to store and to read.
// A complex operator A + iB on u + iv takes three real products instead of four:
//   re = A (u + v) - (A + B) v,   im = A (u + v) + (B - A) u.
// Yukawa's operators are real: two products.
//
// Kernel: one block of 8 warps per tile of 32 pairs of one operator (16 pairs
// where 32 do not fit).  It gathers the tile's inputs, rotates and combines them
// into shared memory once, then streams the operator through a 4-stage cp.async
// ring in chunks of 8 columns; a warp owns 8 pairs and every second (fourth)
// 8-row tile of both blocks, with mma.sync m8n8k4 .f64 (256 FMA per warp
// instruction, the FP64 pipe's full rate).  Rows of the two blocks are numbered
// alike, so the even and odd results of an order meet in one thread; they are
// rotated back, transposed through shared memory and added to the target's
// expansion in whole 256-byte rows.
//
// Bound: the FP64 pipe.  Measured on one B200, M2L phase alone, against dense
// K x K operators of all 316 positions: Laplace FP64 (box tiles, plain FMAs)
// 262,144 clustered points, p = 12, depth 5 (206,548 box pairs) 5.68 -> 0.47 ms;
// 100,000 uniform points, p = 8, depth 4 (640,584 pairs) 1.71 -> 0.44 ms;
// Helmholtz (2K x 2K real form on the same tensor instruction) 1,048,576 sphere
// points, p = 16, depth 5 (291,998 pairs) 7.84 -> 5.22 ms.
#include <cuda_runtime.h>

#include <algorithm>

#include "internal.h"
#include "kernels.h"

namespace fmmb {
namespace {

constexpr int kThreads = 256;
constexpr int kStages = 4;
constexpr int kKC = 8;      // operator columns per chunk
constexpr int kPhiM = 21;   // orders 0..20 of the rotation table

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// MODE 0 Laplace (one real product), 1 Helmholtz (three), 2 Yukawa (one
// operator, two inputs).  NR: 8-row tiles per warp and block; NQ: 8-pair
// groups per tile (4 or 2).
template <int MODE, int NR, int NQ>
__global__ void __launch_bounds__(kThreads) m2l_parity(ParityArgs P) {
  constexpr int NP = 8 * NQ;        // pairs of the block
  constexpr int S = NP + 4;         // input row stride: S mod 16 = 4, the fragment reads hit different banks
  constexpr int NH = 8 / NQ;        // warps sharing a pair group
  constexpr int CX = MODE == 0 ? 1 : 2;     // input components (real, or u and v)
  constexpr int NPROD = MODE == 1 ? 3 : 1;  // operator images streamed one after another
  extern __shared__ __align__(16) double sm[];
  __shared__ int s_src[NP], s_dst[NP], s_phi[NP];
  __shared__ uchar2 s_nm[256];  // row (n, m), m > 0 rows first
  const int p = P.p, E = (p + 1) * (p + 2) / 2, O = p * (p + 1) / 2, K = E + O;
  const int RTE = (E + 7) / 8, RTO = (O + 7) / 8, RSE = 8 * RTE + 4, RSO = 8 * RTO + 4;
  // inputs: even [CX][8 RTE][S], odd [CX][8 RTO][S], then the operator ring
  double* XE = sm;
  double* XO = XE + CX * 8 * RTE * S;
  double* ring = XO + CX * 8 * RTO * S;
  const int tile = blockIdx.x / (4 / NQ), part = blockIdx.x % (4 / NQ);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const double* img = P.img + (size_t)P.tile_cls[tile] * P.img_stride;
  const int nE = NPROD * RTE, nch = nE + NPROD * RTO;  // chunks of the two blocks
  auto issue = [&](int c) {
    if (c < nch) {
      const int RS = c < nE ? RSE : RSO;
      const double* src = img + (c < nE ? (size_t)c * kKC * RSE : (size_t)nE * kKC * RSE + (size_t)(c - nE) * kKC * RSO);
      const uint32_t dst = smem_addr(ring + (size_t)(c % kStages) * kKC * RSE);
      for (int e = tid; e < kKC * RS / 2; e += kThreads)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * e), "l"(src + 2 * e) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int c = 0; c < kStages - 1; c++) issue(c);
  if (tid < NP) {
    const size_t e = (size_t)tile * 32 + part * NP + tid;
    s_src[tid] = P.tile_src[e];
    s_dst[tid] = P.tile_dst[e];
    s_phi[tid] = P.tile_phi[e];
  }
  for (int r = tid; r < E; r += kThreads) {
    int n, m = 0;
    if (r < O) {  // r = n (n - 1) / 2 + m - 1
      n = 1;
      while ((n + 1) * n / 2 <= r) n++;
      m = r - n * (n - 1) / 2 + 1;
    } else {
      n = r - O;
    }
    s_nm[r] = make_uchar2((unsigned char)n, (unsigned char)m);
  }
  __syncthreads();
  // gather: a warp instruction takes 8 rows x 4 pairs (conflict-free stores)
  const int gp = lane & 3, gr = lane >> 2;
  for (int g = warp; g < RTE * (NP / 4); g += kThreads / 32) {
    const int r = 8 * (g / (NP / 4)) + gr, pr = 4 * (g % (NP / 4)) + gp;
    const int src = s_src[pr];
    double e0 = 0, e1 = 0, o0 = 0, o1 = 0;
    if (src >= 0 && r < E) {
      const int n = s_nm[r].x, m = s_nm[r].y;
      if (MODE == 0) {
        const double* x = P.xin + (size_t)src * K + n * n;
        if (m == 0) {
          e0 = x[0];
        } else {
          const double re = x[2 * m - 1], im = x[2 * m];
          const double2 cs = P.phi[s_phi[pr] * kPhiM + m];
          e0 = cs.x * re - cs.y * im;
          o0 = cs.x * im + cs.y * re;
        }
      } else {
        const double* x = P.xin + (size_t)src * 2 * K + n * n + n;
        if (m == 0) {
          e0 = x[0];
          e1 = x[K];
        } else {
          const double ar = x[m], ai = x[K + m], br = x[-m], bi = x[K - m];
          const double2 cs = P.phi[s_phi[pr] * kPhiM + m];
          const double pr_ = cs.x * ar - cs.y * ai, pi_ = cs.x * ai + cs.y * ar;  // E_n^m e^{i m phi}
          const double mr_ = cs.x * br + cs.y * bi, mi_ = cs.x * bi - cs.y * br;  // E_n^-m e^{-i m phi}
          e0 = pr_ + mr_;
          e1 = pi_ + mi_;
          o0 = pr_ - mr_;
          o1 = pi_ - mi_;
        }
      }
    }
    XE[r * S + pr] = e0;
    if (CX == 2) XE[(8 * RTE + r) * S + pr] = e1;
    if (r < 8 * RTO) {
      const bool odd = r < O;
      XO[r * S + pr] = odd ? o0 : 0.0;
      if (CX == 2) XO[(8 * RTO + r) * S + pr] = odd ? o1 : 0.0;
    }
  }
  const int q = warp % NQ, h = warp / NQ, gq = lane >> 2, tq = lane & 3;
  // results of the two blocks: [even / odd][row tile][component][pair parity]
  double acc[2][NR][CX][2];
#pragma unroll
  for (int b = 0; b < 2; b++)
#pragma unroll
    for (int i = 0; i < NR; i++)
#pragma unroll
      for (int x = 0; x < CX; x++) acc[b][i][x][0] = acc[b][i][x][1] = 0.0;
  int c = 0;
#pragma unroll
  for (int b = 0; b < 2; b++) {
    const int RT = b ? RTO : RTE, RS = b ? RSO : RSE;
    const double* X0 = (b ? XO : XE) + 8 * q + gq;
    const double* X1 = X0 + 8 * RT * S;
#pragma unroll
    for (int pd = 0; pd < NPROD; pd++) {
      if (pd == 1) {  // A (u + v) is shared by the two components
#pragma unroll
        for (int i = 0; i < NR; i++) {
          acc[b][i][CX - 1][0] = acc[b][i][0][0];
          acc[b][i][CX - 1][1] = acc[b][i][0][1];
        }
      }
      for (int kc = 0; kc < RT; kc++, c++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();  // chunk c is there (the first: the inputs too); chunk c - 1's stage is free
        issue(c + kStages - 1);
        const double* a = ring + (size_t)(c % kStages) * kKC * RSE + 8 * h + gq;
#pragma unroll
        for (int k4 = 0; k4 < kKC; k4 += 4) {
          const int kr = k4 + tq, col = kc * kKC + kr;
          double x0 = 0, x1 = 0;
          if (MODE == 0) x0 = X0[col * S];
          if (MODE == 1) x0 = pd == 0 ? X0[col * S] + X1[col * S] : pd == 1 ? X1[col * S] : X0[col * S];
          if (MODE == 2) x0 = X0[col * S], x1 = X1[col * S];
#pragma unroll
          for (int i = 0; i < NR; i++) {
            if (h + NH * i < RT) {  // warp-uniform
              const double av = a[kr * RS + 8 * NH * i];
              dmma884(acc[b][i][pd == 2 ? CX - 1 : 0], av, x0);
              if (MODE == 2) dmma884(acc[b][i][CX - 1], av, x1);
            }
          }
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();  // the inputs are consumed: their memory takes the results, [pair][CX K]
  const int KO = CX * K, YS = KO + 1;
  double* Y = sm;
#pragma unroll
  for (int i = 0; i < NR; i++) {
    const int r = 8 * (h + NH * i) + gq;
    if (r >= E) continue;
    const int n = s_nm[r].x, m = s_nm[r].y;
#pragma unroll
    for (int v = 0; v < 2; v++) {
      const int pr = 8 * q + 2 * tq + v;
      if (s_dst[pr] < 0) continue;
      double* y = Y + pr * YS + n * n;
      const double2 cs = P.phi[s_phi[pr] * kPhiM + m];
      const double er = acc[0][i][0][v], orr = acc[1][i][0][v];
      if (MODE == 0) {
        if (m == 0) {
          y[0] = er;
        } else {  // (re + i im) e^{-i m phi}
          y[2 * m - 1] = cs.x * er + cs.y * orr;
          y[2 * m] = cs.x * orr - cs.y * er;
        }
      } else {
        const double ei = acc[0][i][CX - 1][v], oi = acc[1][i][CX - 1][v];
        y += n;
        if (m == 0) {
          y[0] = er;
          y[K] = ei;
        } else {
          const double ar = er + orr, ai = ei + oi, br = er - orr, bi = ei - oi;
          y[m] = cs.x * ar + cs.y * ai;
          y[K + m] = cs.x * ai - cs.y * ar;
          y[-m] = cs.x * br - cs.y * bi;
          y[K - m] = cs.x * bi + cs.y * br;
        }
      }
    }
  }
  __syncthreads();
  for (int pr = warp; pr < NP; pr += kThreads / 32) {
    const int d = s_dst[pr];
    if (d < 0) continue;
    double* o = P.out + (size_t)d * KO;
    for (int k = lane; k < KO; k += 32) atomicAdd(o + k, Y[pr * YS + k]);
  }
}

struct Shape {
  int RTE, RTO, CX, NQ;
  size_t smem;
};
Shape shape(int mode, int p) {
  Shape s;
  s.RTE = ((p + 1) * (p + 2) / 2 + 7) / 8;
  s.RTO = (p * (p + 1) / 2 + 7) / 8;
  s.CX = mode == 0 ? 1 : 2;
  for (s.NQ = 4;; s.NQ = 2) {  // 16 pairs where the inputs of 32 do not fit (complex, p > 16)
    s.smem = ((size_t)s.CX * 8 * (s.RTE + s.RTO) * (8 * s.NQ + 4) + (size_t)kStages * kKC * (8 * s.RTE + 4)) * sizeof(double);
    if (s.NQ == 2 || s.smem <= 224 * 1024) return s;
  }
}

template <typename F>
void with_kernel(int mode, int p, F f) {
  const Shape s = shape(mode, p);
  const int nr = (s.RTE + 8 / s.NQ - 1) / (8 / s.NQ);
  auto rows = [&](auto m, auto q) {
    constexpr int M = decltype(m)::value, Q = decltype(q)::value;
    if (nr <= 3) f(m2l_parity<M, 3, Q>, s);
    else if (nr <= 5) f(m2l_parity<M, 5, Q>, s);
    else if (nr <= 6) f(m2l_parity<M, 6, Q>, s);
    else if (nr <= 8) f(m2l_parity<M, 8, Q>, s);
    else if (Q == 4 && nr <= 10) f(m2l_parity<M, Q == 4 ? 10 : 8, Q>, s);
    else if (M == 0) f(m2l_parity<M, M == 0 ? 15 : 8, Q>, s);
    else throw Error{FMMB_ERR_ARG, "order too high for the FP64 M2L"};
  };
  using I0 = std::integral_constant<int, 0>;
  using I1 = std::integral_constant<int, 1>;
  using I2 = std::integral_constant<int, 2>;
  using I4 = std::integral_constant<int, 4>;
  if (mode == 0) rows(I0{}, I4{});
  else if (mode == 1 && s.NQ == 4) rows(I1{}, I4{});
  else if (mode == 1) rows(I1{}, I2{});
  else if (s.NQ == 4) rows(I2{}, I4{});
  else rows(I2{}, I2{});
}

}  // namespace

// doubles of one operator: the images of the even block, then of the odd one,
// each [column, padded to 8][row, padded to 8 and 4 more]
size_t parity_img_stride(int mode, int p) {
  const Shape s = shape(mode, p);
  return (mode == 1 ? 3 : 1) * ((size_t)8 * s.RTE * (8 * s.RTE + 4) + (size_t)8 * s.RTO * (8 * s.RTO + 4));
}

void prepare_m2l_parity(int mode, int p) {
  with_kernel(mode, p, [](auto k, const Shape& s) {
    FMMB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.smem));
  });
}

void launch_m2l_parity(int mode, const ParityArgs& a, cudaStream_t st) {
  if (a.ntile <= 0) return;
  with_kernel(mode, a.p, [&](auto k, const Shape& s) {
    k<<<(unsigned)(a.ntile * (4 / s.NQ)), kThreads, s.smem, st>>>(a);
  });
  FMMB_CHECK_LAUNCH();
}

}  // namespace fmmb
