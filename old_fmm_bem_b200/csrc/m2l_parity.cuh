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
// Kernel, one instance per order: a block per tile of 32 pairs of one operator
// (16 pairs where 32 do not fit).  It gathers the tile's inputs, rotates and
// combines them into shared memory once, then streams the operator through a
// 4-slot ring of bulk copies in chunks of 8 columns: the warps wait for a chunk
// and free its slot through mbarriers, without block barriers between chunks, and
// take turns at waiting for a free slot and sending for the next chunk (the same
// warp each time fell behind and held the others up; a warp of its own for it
// left 96 registers a thread and spilled).  A warp owns 8 pairs and every second
// (fourth, eighth) 8-row tile of both blocks, with mma.sync m8n8k4 .f64 (256 FMA
// per warp instruction, the FP64 pipe's full rate).  Columns k, k + 4
// of a chunk lie side by side, operator and inputs alike, so that one 16-byte
// read feeds two MMAs.  Rows of the two blocks are numbered alike, so the even
// and odd results of an order meet in one thread; they are rotated back,
// transposed through shared memory and added to the target's expansion in
// whole 256-byte rows.  8 warps where two or more blocks fit an SM, 16 where
// one does.
//
// Bound: the FP64 pipe.  Measured on one B200, M2L phase alone, against dense
// K x K operators of all 316 positions: Laplace FP64 (box tiles, plain FMAs)
// 262,144 clustered points, p = 12, depth 5 (206,548 box pairs) 5.68 -> 0.31 ms;
// 100,000 uniform points, p = 8, depth 4 (640,584 pairs) 1.71 -> 0.37 ms;
// Helmholtz (2K x 2K real form on the same tensor instruction) 1,048,576 sphere
// points, p = 16, depth 5 (291,998 pairs) 7.84 -> 3.68 ms (4.13
// with one warp sending for every chunk)
// (8 instead of 16 warps where one block fills an SM: 5.22 ms, too few per
// scheduler to hide the tensor instruction's and the shared-memory reads'
// latency).
#pragma once

#include <cuda_runtime.h>

#include "internal.h"
#include "kernels.h"

namespace fmmb {
namespace parity {

constexpr int kStages = 4, kLead = 2;  // ring slots; chunks copied ahead of the one in use
constexpr int kKC = 8;      // operator columns per chunk
constexpr int kPhiM = 21;   // orders 0..20 of the rotation table

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// A wait is bounded: the thread is suspended up to kSuspendNs per try, kSpinLimit
// tries (seconds); a timeout sets the plan's device error code.
constexpr unsigned kSpinLimit = 1u << 18, kSuspendNs = 16384;
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  const uint32_t a = smem_addr(bar);
  for (unsigned it = 0; it < kSpinLimit; it++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(a), "r"(parity), "n"(kSuspendNs)
        : "memory");
    if (done) return true;
  }
  return false;
}
// bulk copy of `bytes` (a multiple of 16) to shared memory, completing on bar
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}

// Sizes of an instance.  MODE 0 Laplace (one real product), 1 Helmholtz
// (three), 2 Yukawa (one operator, two inputs).
template <int MODE, int P>
struct Cfg {
  static constexpr int E = (P + 1) * (P + 2) / 2, O = P * (P + 1) / 2, K = E + O;
  static constexpr int RTE = parity_tiles(E), RTO = parity_tiles(O);  // 8-row tiles (and 8-column chunks) of a block
  static constexpr int RSE = parity_row(RTE), RSO = parity_row(RTO);
  static constexpr int CX = MODE == 0 ? 1 : 2;     // input components (real, or u and v)
  static constexpr int NPROD = MODE == 1 ? 3 : 1;  // operator images streamed one after another
  static constexpr size_t smem(int nq) {
    return ((size_t)CX * 8 * (RTE + RTO) * (8 * nq + 2) + (size_t)kStages * kKC * RSE) * sizeof(double);
  }
  static constexpr int NQ = smem(4) <= 224 * 1024 ? 4 : 2;  // 8-pair groups per tile
  static constexpr size_t kSmem = smem(NQ);
  static constexpr int NW = 2 * kSmem + 4096 > 227 * 1024 ? 16 : 8;  // warps: two blocks per SM, or one
  static constexpr int NP = 8 * NQ;                                  // pairs of the block
  static constexpr int S = NP + 2;    // input row stride (pairs of columns): S mod 8 = 2, conflict-free 16-byte reads
  static constexpr int NH = NW / NQ;  // warps sharing a pair group
  static constexpr int NR = (RTE + NH - 1) / NH;  // 8-row tiles per warp and block
};

// One column chunk of one block: the warp's row tiles against its 8 pairs.
// PD: which product of the complex form.
template <int MODE, int PD, int RT, int RS, int S, int NH, int NR, int CX>
__device__ __forceinline__ void chunk(const double2* a, const double2* X, int h, double (&acc)[NR][CX][2]) {
  constexpr int CS = RT * 4 * S;  // from component u to v
  double2 x0, x1;
  if (MODE == 1 && PD == 0) {
    const double2 u = X[0], v = X[CS];
    x0 = make_double2(u.x + v.x, u.y + v.y);
  } else if (MODE == 1 && PD == 1) {
    x0 = X[CS];
  } else {
    x0 = X[0];
    if (MODE == 2) x1 = X[CS];
  }
  double2 av[NR];
#pragma unroll
  for (int i = 0; i < NR; i++)
    if (NH * i + NH - 1 < RT || h + NH * i < RT) av[i] = a[8 * NH * i];  // warp-uniform; only the last tiles are tested
  constexpr int T = MODE == 1 && PD == 2 ? CX - 1 : 0;
#pragma unroll
  for (int k = 0; k < 2; k++)  // columns k, k + 4: an accumulator's two MMAs stand NR apart
#pragma unroll
    for (int i = 0; i < NR; i++) {
      if (NH * i + NH - 1 < RT || h + NH * i < RT) {
        dmma884(acc[i][T], k ? av[i].y : av[i].x, k ? x0.y : x0.x);
        if (MODE == 2) dmma884(acc[i][CX - 1], k ? av[i].y : av[i].x, k ? x1.y : x1.x);
      }
    }
}

template <int MODE, int P>
__global__ void __launch_bounds__(Cfg<MODE, P>::NW * 32) m2l_parity(ParityArgs A) {
  using C = Cfg<MODE, P>;
  constexpr int E = C::E, O = C::O, K = C::K, RTE = C::RTE, RTO = C::RTO, RSE = C::RSE, RSO = C::RSO, CX = C::CX;
  constexpr int NP = C::NP, S = C::S, NH = C::NH, NR = C::NR, kThreads = C::NW * 32;
  extern __shared__ __align__(16) double sm[];
  __shared__ int s_src[NP], s_dst[NP], s_phi[NP];
  __shared__ uchar2 s_nm[E];  // row (n, m), m > 0 rows first
  __shared__ uint64_t full[kStages], empty[kStages];
  __shared__ int s_fail;
  // inputs: even [CX][RTE][4][S] column pairs (k, k + 4), odd [CX][RTO][4][S], then the operator ring
  double* XE = sm;
  double* XO = XE + CX * 8 * RTE * S;
  double* ring = XO + CX * 8 * RTO * S;
  const int tile = blockIdx.x / (4 / C::NQ), part = blockIdx.x % (4 / C::NQ);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const double* img = A.img + (size_t)A.tile_cls[tile] * A.img_stride;
  constexpr int nE = C::NPROD * RTE, nch = nE + C::NPROD * RTO;  // chunks of the two blocks
  int sent = -1;  // the last chunk this thread sent for
  // copies chunk c into its slot once every warp is done with chunk c - kStages
  auto issue = [&](int c) {
    if (c >= nch) return true;
    if (c >= kStages && !mbar_wait(&empty[c % kStages], (c / kStages - 1) & 1)) return false;
    const double* src = img + (c < nE ? (size_t)c * kKC * RSE : (size_t)nE * kKC * RSE + (size_t)(c - nE) * kKC * RSO);
    sent = c;
    bulk_g2s(ring + (size_t)(c % kStages) * kKC * RSE, src, (c < nE ? RSE : RSO) * kKC * 8, &full[c % kStages]);
    return true;
  };
  if (tid == 0) {
    for (int i = 0; i < kStages; i++) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], C::NW);
    }
    s_fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int c = 0; c < kLead; c++) issue(c);
  }
  if (tid < NP) {
    const size_t e = (size_t)tile * 32 + part * NP + tid;
    s_src[tid] = A.tile_src[e];
    s_dst[tid] = A.tile_dst[e];
    s_phi[tid] = A.tile_phi[e];
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
  // gather: a warp instruction takes 8 rows (one chunk of columns) x 4 pairs
  const int gp = lane & 3, gr = lane >> 2;
  for (int g = warp; g < RTE * (NP / 4); g += C::NW) {
    const int kc = g / (NP / 4), r = 8 * kc + gr, pr = 4 * (g % (NP / 4)) + gp;
    const int src = s_src[pr];
    double e0 = 0, e1 = 0, o0 = 0, o1 = 0;
    if (src >= 0 && r < E) {
      const int n = s_nm[r].x, m = s_nm[r].y;
      if (MODE == 0) {
        const double* x = A.xin + (size_t)src * K + n * n;
        if (m == 0) {
          e0 = x[0];
        } else {
          const double re = x[2 * m - 1], im = x[2 * m];
          const double2 cs = A.phi[s_phi[pr] * kPhiM + m];
          e0 = cs.x * re - cs.y * im;
          o0 = cs.x * im + cs.y * re;
        }
      } else {
        const double* x = A.xin + (size_t)src * 2 * K + n * n + n;
        if (m == 0) {
          e0 = x[0];
          e1 = x[K];
        } else {
          const double ar = x[m], ai = x[K + m], br = x[-m], bi = x[K - m];
          const double2 cs = A.phi[s_phi[pr] * kPhiM + m];
          const double pr_ = cs.x * ar - cs.y * ai, pi_ = cs.x * ai + cs.y * ar;  // E_n^m e^{i m phi}
          const double mr_ = cs.x * br + cs.y * bi, mi_ = cs.x * bi - cs.y * br;  // E_n^-m e^{-i m phi}
          e0 = pr_ + mr_;
          e1 = pi_ + mi_;
          o0 = pr_ - mr_;
          o1 = pi_ - mi_;
        }
      }
    }
    const int at = ((4 * kc + (gr & 3)) * S + pr) * 2 + (gr >> 2);
    XE[at] = e0;
    if (CX == 2) XE[8 * RTE * S + at] = e1;
    if (kc < RTO) {
      const bool odd = r < O;
      XO[at] = odd ? o0 : 0.0;
      if (CX == 2) XO[8 * RTO * S + at] = odd ? o1 : 0.0;
    }
  }
  const int q = warp % C::NQ, h = warp / C::NQ, gq = lane >> 2, tq = lane & 3;
  double acE[NR][CX][2], acO[NR][CX][2];  // results of the two blocks: [row tile][component][pair parity]
#pragma unroll
  for (int i = 0; i < NR; i++)
#pragma unroll
    for (int x = 0; x < CX; x++) acE[i][x][0] = acE[i][x][1] = acO[i][x][0] = acO[i][x][1] = 0.0;
  __syncthreads();  // the inputs are in place
  int c = 0;
  bool ok = true;
  // one product of one block: RT chunks of columns
  auto product = [&](auto pd, auto rt, const double* X, auto& acc) {
    constexpr int PD = decltype(pd)::value, RT = decltype(rt)::value, RS = parity_row(RT);
    const double2* x = reinterpret_cast<const double2*>(X) + tq * S + 8 * q + gq;
    if (PD == 1) {  // A (u + v) is shared by the two components
#pragma unroll
      for (int i = 0; i < NR; i++) {
        acc[i][CX - 1][0] = acc[i][0][0];
        acc[i][CX - 1][1] = acc[i][0][1];
      }
    }
    for (int kc = 0; kc < RT && ok; kc++, c++, x += 4 * S) {
      if (warp == c % C::NW && lane == 0) ok = issue(c + kLead);  // the warps take turns
      ok = mbar_wait(&full[c % kStages], (c / kStages) & 1) && ok;
      if (!__all_sync(0xffffffffu, ok)) {
        ok = false;
        s_fail = 1;
        break;
      }
      const double2* a = reinterpret_cast<const double2*>(ring + (size_t)(c % kStages) * kKC * RSE) + tq * RS + 8 * h + gq;
      chunk<MODE, PD, RT, RS, S, NH, NR, CX>(a, x, h, acc);
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[c % kStages]);
    }
  };
  using I0 = std::integral_constant<int, 0>;
  using I1 = std::integral_constant<int, 1>;
  using I2 = std::integral_constant<int, 2>;
  using TE = std::integral_constant<int, RTE>;
  using TO = std::integral_constant<int, RTO>;
  product(I0{}, TE{}, XE, acE);
  if (MODE == 1) {
    product(I1{}, TE{}, XE, acE);
    product(I2{}, TE{}, XE, acE);
  }
  product(I0{}, TO{}, XO, acO);
  if (MODE == 1) {
    product(I1{}, TO{}, XO, acO);
    product(I2{}, TO{}, XO, acO);
  }
  __syncthreads();  // the inputs are consumed: their memory takes the results, [pair][CX K]
  if (s_fail) {  // a wait timed out: let the copies in flight land, report, leave
    if (sent >= 0) mbar_wait(&full[sent % kStages], (sent / kStages) & 1);
    if (tid == 0) {
      for (int i = 0; i < kLead; i++) mbar_wait(&full[i], 0);
      atomicExch(A.err, 100);
    }
    return;
  }
  constexpr int KO = CX * K, YS = KO + 1;
  static_assert(NP * YS <= CX * 8 * (RTE + RTO) * S, "results in the inputs' memory");
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
      const double2 cs = A.phi[s_phi[pr] * kPhiM + m];
      const double er = acE[i][0][v], orr = acO[i][0][v];
      if (MODE == 0) {
        if (m == 0) {
          y[0] = er;
        } else {  // (re + i im) e^{-i m phi}
          y[2 * m - 1] = cs.x * er + cs.y * orr;
          y[2 * m] = cs.x * orr - cs.y * er;
        }
      } else {
        const double ei = acE[i][CX - 1][v], oi = acO[i][CX - 1][v];
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
  for (int pr = warp; pr < NP; pr += C::NW) {
    const int d = s_dst[pr];
    if (d < 0) continue;
    double* o = A.out + (size_t)d * KO;
    for (int k = lane; k < KO; k += 32) atomicAdd(o + k, Y[pr * YS + k]);
  }
}

template <int MODE, int P>
void run(int p, const ParityArgs* a, cudaStream_t st) {
  if constexpr (P > 20) {
    throw Error{FMMB_ERR_ARG, "order too high for the FP64 M2L"};
  } else {
    using C = Cfg<MODE, P>;
    if (p != P) return run<MODE, P + 1>(p, a, st);
    if (a)
      m2l_parity<MODE, P><<<(unsigned)(a->ntile * (4 / C::NQ)), C::NW * 32, C::kSmem, st>>>(*a);
    else
      FMMB_CUDA(cudaFuncSetAttribute(m2l_parity<MODE, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::kSmem));
  }
}

}  // namespace parity
}  // namespace fmmb
