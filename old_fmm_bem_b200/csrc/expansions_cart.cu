// P2M and L2P from Cartesian solid-harmonic recurrences (accurate semantics).
//
// The reference evaluates r^n fac(n,m) P_n^m(cos a) e^{-i m b} through
// spherical angles (acos, atan, exp; kernel/multipole.cxx:7-35,
// kernel/G_p2m.cxx:28-55) and the local-expansion gradient through spherical
// derivatives with a 1/sin(theta) (kernel/G_l2p.cxx:44-70).  In exact
// arithmetic the same quantities follow from the homogeneous polynomials
//   S_n^m(x) = r^n P_n^m(cos theta) e^{i m phi}   (Condon-Shortley phase)
// without any trigonometric function:
//   S_m^m = -(2m-1) (x + i y) S_{m-1}^{m-1},   S_{m+1}^m = (2m+1) z S_m^m,
//   (n-m) S_n^m = (2n-1) z S_{n-1}^m - (n+m-1) r^2 S_{n-2}^m,
// with the ladder identities
//   d/dz S_n^m = (n+m) S_{n-1}^m,  (d/dx + i d/dy) S_n^m = S_{n-1}^{m+1},
//   (d/dx - i d/dy) S_n^m = -(n+m)(n+m-1) S_{n-1}^{m-1},
//   S_{n}^{-1} = -conj(S_n^1) / (n (n+1)).
// Multipole basis: fac(n,m) conj(S_n^m); local evaluation: Re sum w_m
// fac(n,m) L_n^m S_n^m with w_0 = 1, w_m = 2.  This form has no singular
// points (a target on a box axis or at a box centre is fine), so it is used
// for accurate semantics; reference semantics keep the spherical kernels
// of kernels_fp64.cu, which reproduce the reference's eps-shifted radius and
// single-precision angles.
#include <cuda_runtime.h>

#include <cmath>

#include "internal.h"
#include "kernels.h"

namespace fmmb {
namespace {

struct cplx {
  double re, im;
};

// 1/k for the Legendre-type recurrences (k = n - m <= 40): avoids FP64 divides
__constant__ double c_inv[41] = {0.0,      1.0 / 1,  1.0 / 2,  1.0 / 3,  1.0 / 4,  1.0 / 5,  1.0 / 6,  1.0 / 7,
                                 1.0 / 8,  1.0 / 9,  1.0 / 10, 1.0 / 11, 1.0 / 12, 1.0 / 13, 1.0 / 14, 1.0 / 15,
                                 1.0 / 16, 1.0 / 17, 1.0 / 18, 1.0 / 19, 1.0 / 20, 1.0 / 21, 1.0 / 22, 1.0 / 23,
                                 1.0 / 24, 1.0 / 25, 1.0 / 26, 1.0 / 27, 1.0 / 28, 1.0 / 29, 1.0 / 30, 1.0 / 31,
                                 1.0 / 32, 1.0 / 33, 1.0 / 34, 1.0 / 35, 1.0 / 36, 1.0 / 37, 1.0 / 38, 1.0 / 39,
                                 1.0 / 40};
// Recurrence of A_n^m (below): A_n = alpha z A_{n-1} - beta r^2 A_{n-2}, alpha =
// (2n-1)/(n-m), beta = (n+m-1)/(n-m), at n (n+1) / 2 + m
struct RecTab {
  double2 d[231];
  constexpr RecTab() : d() {
    for (int n = 0; n <= 20; n++)
      for (int m = 0; m < n; m++) {
        d[n * (n + 1) / 2 + m].x = (2.0 * n - 1.0) / (n - m);
        d[n * (n + 1) / 2 + m].y = (n + m - 1.0) / (n - m);
      }
  }
  __device__ const double2& operator[](int i) const { return d[i]; }
};
__constant__ RecTab c_rec = RecTab();
// The FP32 kernels write S_n^m = g_n^m B_n^m t^m, t = x + i y, with the monic recurrence
//   B_m = 1,  B_n = z B_{n-1} - c_n r^2 B_{n-2},  c_n = (n+m-1)(n-m-1) / ((2n-1)(2n-3)):
// three operations a term, the factors g taken up by the coefficients.
// g_n^m = (-1)^m (2m-1)!! prod_{k=m+1..n} (2k-1)/(k-m), at n (n+1) / 2 + m
struct MonicTab {
  double g[231];
  constexpr MonicTab() : g() {
    double f = 1.0;  // (-1)^m (2m-1)!!
    for (int m = 0; m <= 20; m++) {
      if (m > 0) f *= -(2.0 * m - 1.0);
      double v = f;
      for (int n = m; n <= 20; n++) {
        if (n > m) v *= (2.0 * n - 1.0) / (n - m);
        g[n * (n + 1) / 2 + m] = v;
      }
    }
  }
};
__constant__ MonicTab c_monic = MonicTab();

__device__ constexpr float monic_c(int n, int m) {  // c_n, n > m
  return n > m + 1 ? (float)((double)((n + m - 1) * (n - m - 1)) / (double)((2 * n - 1) * (2 * n - 3))) : 0.f;
}
__device__ __forceinline__ cplx cmul(cplx a, cplx b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
__device__ __forceinline__ cplx cscale(cplx a, double s) { return {a.re * s, a.im * s}; }

__device__ __forceinline__ void box_center(int key, float xmin, float ymin, float zmin, double rb, double& xc, double& yc,
                                           double& zc) {
  int cx = 0, cy = 0, cz = 0;
  for (int i = 0; i < 10; i++) {
    cy |= ((key >> (3 * i)) & 1) << i;
    cx |= ((key >> (3 * i + 1)) & 1) << i;
    cz |= ((key >> (3 * i + 2)) & 1) << i;
  }
  xc = (double)xmin + (cx + 0.5) * rb;
  yc = (double)ymin + (cy + 0.5) * rb;
  zc = (double)zmin + (cz + 0.5) * rb;
}

// ------------------------------------------------------------------ P2M
// One block (4 warps) per source leaf, 128 points at a time.  With
//   S_n^m = A_n^m s_m,  s_m = -(2m-1) (x + i y) s_{m-1},  A_m^m = 1 and A real,
//   (n-m) A_n^m = (2n-1) z A_{n-1}^m - (n+m-1) r^2 A_{n-2}^m,
// the sums over the points are, for each order m, a product of the real
// (p + 1 - m) x points matrix A with a points x NCOL one (w s_m, real and
// imaginary parts), done on the FP64 tensor instruction: every warp takes orders
// of its own (dealt so that all have about the same number of terms), evaluates
// the column of A for 32 points at a time, one a lane, and multiplies.  Charges
// take one complex w = q; dipoles three, ((n_x - i n_y) / 2, (n_x + i n_y) / 2,
// n_z) q, whose sums U_1..U_3 give by the ladder identities
//   n . grad S_n^m: U_1[n-1, m+1] - (n+m)(n+m-1) U_2[n-1, m-1] + (n+m) U_3[n-1, m].
// Reference semantics take the same sums with the reference's angles and
// eps-shifted radius (kernel/G_p2m.cxx:28-55) in place of the coordinates.
// Bound: the FP64 pipe (a quarter of the tensor instruction's columns hold a
// charge's sums).  One lane per order and a shared-memory sum per term before:
// 262,144 clustered points, p = 12: 0.93 ms; 0.19 now.
constexpr int kPts = 128;
constexpr int kPS = 36;     // row stride of a warp's staging: 32 points, conflict-free fragment reads
constexpr int kRows = 24;   // orders' columns: up to 21 rows in tiles of 8

__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// the reference's azimuth (kernel/G_p2m.cxx:33-41), coordinates relative to the box centre
__device__ __forceinline__ double ref_azimuth(double x, double y, const Sem& s) {
  if (fabs(x) + fabs(y) < s.ang_eps) return 0.0;
  if (fabs(x) < s.ang_eps) return y / fabs(y) * s.pi_ang * 0.5;
  if (x > 0) return atan(y / x);
  return atan(y / x) + s.pi_ang;
}

template <int KER, bool REF>
__global__ void __launch_bounds__(kPts) p2m_dmma(int p, int K, const int* __restrict__ keys, const int2* __restrict__ leaf,
                                                const float4* __restrict__ spos, const float4* __restrict__ snrm,
                                                const float* __restrict__ qs, const double* __restrict__ fac, Sem sem,
                                                float xmin, float ymin, float zmin, double rb, double* __restrict__ M) {
  constexpr bool DIP = KER == FMMB_LAPLACE_GNJ;
  constexpr int NCOL = DIP ? 6 : 2;
  extern __shared__ double sm[];
  const int NT = (p + 1) * (p + 2) / 2, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gq = lane >> 2, tq = lane & 3;
  double* sum = sm;                                              // [terms, by order][NCOL]
  double* mine = sum + NCOL * NT + warp * (kRows + NCOL) * kPS;  // the warp's columns of A and w s_m
  double* wq = mine + kRows * kPS;
  for (int c = threadIdx.x; c < NCOL * NT; c += kPts) sum[c] = 0.0;
  __syncthreads();
  const int b = blockIdx.x;
  double xc, yc, zc;
  box_center(keys[b], xmin, ymin, zmin, rb, xc, yc, zc);
  const int2 lf = leaf[b];
  const double inv_rb = 1.0 / rb;
  for (int base = 0; base < lf.y; base += kPts) {
    const int nch = min(kPts, lf.y - base + 31) / 32;  // groups of 32 points, one point of each a lane
    double x[4], y[4], z[4], r2[4], sr[4], si[4], w[4][DIP ? 3 : 1];
#pragma unroll
    for (int ch = 0; ch < 4; ch++) {
      const int i = base + 32 * ch + lane;
      const bool on = i < lf.y;
      const int j = lf.x + (on ? i : 0);
      const float4 v = spos[j];
      const float q = on ? qs[j] : 0.f;
      const double dx = (double)v.x - xc, dy = (double)v.y - yc, dz = (double)v.z - zc;
      if (REF) {
        const double rh = sqrt(dx * dx + dy * dy + dz * dz) + sem.rho_eps;
        const double al = rh == 0.0 ? 0.0 : acos(dz / rh);
        double sb, cb;
        sincos(ref_azimuth(dx, dy, sem), &sb, &cb);
        const double rs = rh / rb, xx = cos(al), s2 = sqrt((1 - xx) * (1 + xx));
        x[ch] = rs * s2 * cb;
        y[ch] = rs * s2 * sb;
        z[ch] = rs * xx;
        r2[ch] = rs * rs;
      } else {
        x[ch] = dx * inv_rb;
        y[ch] = dy * inv_rb;
        z[ch] = dz * inv_rb;
        r2[ch] = x[ch] * x[ch] + y[ch] * y[ch] + z[ch] * z[ch];
      }
      if (DIP) {
        const float4 n = snrm[j];
        w[ch][0] = 0.5 * ((double)(q * n.x) * inv_rb);
        w[ch][DIP ? 1 : 0] = 0.5 * ((double)(q * n.y) * inv_rb);
        w[ch][DIP ? 2 : 0] = (double)(q * n.z) * inv_rb;
      } else {
        w[ch][0] = (double)q;
      }
      sr[ch] = 1.0;
      si[ch] = 0.0;
    }
    int row0 = 0;
    for (int m = 0; m <= p; row0 += p + 1 - m, m++) {
      if (m > 0) {
        const double f = -(2.0 * m - 1.0);
#pragma unroll
        for (int ch = 0; ch < 4; ch++) {
          const double t = f * (sr[ch] * x[ch] - si[ch] * y[ch]);
          si[ch] = f * (sr[ch] * y[ch] + si[ch] * x[ch]);
          sr[ch] = t;
        }
      }
      if (((m & 4) ? 3 - (m & 3) : (m & 3)) != warp) continue;  // another warp's order
      double acc[3][2] = {};
      const int nrow = p + 1 - m;
#pragma unroll
      for (int ch = 0; ch < 4; ch++) {
        if (ch >= nch) break;
        __syncwarp();  // the previous group's reads are done
        double a1 = 1.0, a2 = 0.0;
        mine[lane] = 1.0;
        for (int n = m + 1; n <= p; n++) {
          const double2 ab = c_rec[n * (n + 1) / 2 + m];
          const double a = fma(ab.x * z[ch], a1, -(ab.y * r2[ch]) * a2);
          a2 = a1;
          a1 = a;
          mine[(n - m) * kPS + lane] = a;
        }
        if (DIP) {
          const double cx = w[ch][0], cy = w[ch][DIP ? 1 : 0], cz = w[ch][DIP ? 2 : 0];
          wq[lane] = cx * sr[ch] + cy * si[ch];  // (n_x - i n_y) / 2
          wq[kPS + lane] = cx * si[ch] - cy * sr[ch];
          wq[2 * kPS + lane] = cx * sr[ch] - cy * si[ch];  // (n_x + i n_y) / 2
          wq[3 * kPS + lane] = cx * si[ch] + cy * sr[ch];
          wq[4 * kPS + lane] = cz * sr[ch];
          wq[5 * kPS + lane] = cz * si[ch];
        } else {
          wq[lane] = w[ch][0] * sr[ch];
          wq[kPS + lane] = w[ch][0] * si[ch];
        }
        __syncwarp();
#pragma unroll
        for (int k4 = 0; k4 < 32; k4 += 4) {
          const double bf = gq < NCOL ? wq[gq * kPS + k4 + tq] : 0.0;
#pragma unroll
          for (int rt = 0; rt < 3; rt++)
            if (8 * rt < nrow) dmma884(acc[rt], mine[(8 * rt + gq) * kPS + k4 + tq], bf);
        }
      }
      if (2 * tq < NCOL) {
#pragma unroll
        for (int rt = 0; rt < 3; rt++)
          if (8 * rt + gq < nrow) {
            sum[NCOL * (row0 + 8 * rt + gq) + 2 * tq] += acc[rt][0];
            sum[NCOL * (row0 + 8 * rt + gq) + 2 * tq + 1] += acc[rt][1];
          }
      }
    }
  }
  __syncthreads();
  auto U = [&](int n, int m, int u) -> cplx {
    if (m < 0 || m > n) return {0.0, 0.0};
    const double* s = sum + NCOL * (m * (p + 1) - m * (m - 1) / 2 + n - m) + 2 * u;
    return {s[0], s[1]};
  };
  for (int idx = threadIdx.x; idx < NT; idx += kPts) {
    int n = 0;
    while ((n + 1) * (n + 2) / 2 <= idx) n++;
    const int m = idx - n * (n + 1) / 2;
    const double f = fac[ifull_d(n, m)];
    cplx v = {0.0, 0.0};
    if (!DIP) {
      v = U(n, m, 0);
    } else if (n > 0) {
      const cplx up = U(n - 1, m + 1, 0), md = U(n - 1, m, DIP ? 2 : 0);
      const cplx dn = m == 0 ? cplx{up.re, -up.im} : U(n - 1, m - 1, DIP ? 1 : 0);
      const double cm = m == 0 ? 1.0 : -(double)(n + m) * (double)(n + m - 1);
      v = {up.re + cm * dn.re + (n + m) * md.re, up.im + cm * dn.im + (n + m) * md.im};
    }
    double* o = M + (size_t)b * K + n * n;
    if (m == 0) {
      o[0] = f * v.re;
    } else {
      o[2 * m - 1] = f * v.re;
      o[2 * m] = -f * v.im;
    }
  }
}

// ------------------------------------------------------------------ P2M (FP32), charges
// The mixed form's P2M of charges: the sums of p2m_dmma in FP32 and the monic form
// (c_monic), one warp per work item of up to kP2MItem = 64 sources of a leaf.  A
// lane evaluates two points side by side in the two-lane FP32 instructions and
// leaves the columns of consecutive orders in shared memory until they fill 16
// rows; then lane (row, re / im) adds its row over the points.  FP32 terms and
// sums over one item's points; a leaf of several items (the dense leaves of
// clustered points) is summed in FP64 by atomics into zeroed rows.
// Bound: issue slots, the rows' sums (64 shared-memory reads and as many FMAs per
// 16 rows) above the recurrences; 7 KB of shared memory a warp.  (One thread per
// point with all (p+1)^2 terms staged, 43 KB per 64 points: 1,048,576 clustered
// points, p = 12: 0.150 ms; 0.087 now.)
constexpr int kFP = kP2MItem + 4;  // row stride of the staging (floats)
constexpr int kFRows = 16, kFOrders = 5;  // staged rows; orders they span at most (1 + ... + 5 = 15)
constexpr int kFWarps = 4;

template <int P>
__global__ void __launch_bounds__(32 * kFWarps) p2m_f32_charges(int p, int K, int nwork, const int2* __restrict__ work,
                                                                const int* __restrict__ keys, const int2* __restrict__ leaf,
                                                                const float4* __restrict__ spos,
                                                                const float* __restrict__ qs,
                                                                const double* __restrict__ fac, float xmin, float ymin,
                                                                float zmin, double rb, double* __restrict__ M) {
  __shared__ __align__(16) float sA[kFWarps][kFRows][kFP], sW[kFWarps][2 * kFOrders][kFP];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int item = blockIdx.x * kFWarps + warp;
  if (item >= nwork) return;
  const int2 wk = work[item];
  const int b = wk.x;
  double xc, yc, zc;
  box_center(keys[b], xmin, ymin, zmin, rb, xc, yc, zc);
  const int2 lb = leaf[b];
  const bool shared_leaf = lb.y > kP2MItem;  // summed by several items
  const int first = lb.x + wk.y, cnt = min(kP2MItem, lb.y - wk.y);
  const double inv_rb = 1.0 / rb;
  float px[2], py[2], pz[2], pq[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {  // the lane's points 2 lane, 2 lane + 1
    const bool on = 2 * lane + h < cnt;
    const int j = first + (on ? 2 * lane + h : 0);
    const float4 v = spos[j];
    pq[h] = on ? qs[j] : 0.f;
    px[h] = (float)(((double)v.x - xc) * inv_rb);
    py[h] = (float)(((double)v.y - yc) * inv_rb);
    pz[h] = (float)(((double)v.z - zc) * inv_rb);
  }
  const float2 x = make_float2(px[0], px[1]), y = make_float2(py[0], py[1]), z = make_float2(pz[0], pz[1]);
  const float2 nx = make_float2(-px[0], -px[1]), ny = make_float2(-py[0], -py[1]);
  const float2 mr2 = __ffma2_rn(nx, x, __ffma2_rn(ny, y, __fmul2_rn(make_float2(-pz[0], -pz[1]), z)));  // -r^2
  float2 tr = make_float2(pq[0], pq[1]), ti = make_float2(0.f, 0.f);  // q t^m
  int rows = 0, m0 = 0;  // staged rows: the columns n = m..P of orders m0, m0 + 1, ... (constants once unrolled)
  auto flush = [&](int nrow, int ma) {  // lane (row, component) adds its row over the points
    __syncwarp();
    const int r = lane >> 1, c = lane & 1;
    if (r < nrow) {
      int mm = ma, k0 = r;
      while (k0 > P - mm) {
        k0 -= P + 1 - mm;
        mm++;
      }
      const int nn = mm + k0;
      const float4* ar = reinterpret_cast<const float4*>(sA[warp][r]);
      const float4* wr = reinterpret_cast<const float4*>(sW[warp][2 * (mm - ma) + c]);
      float2 a0 = make_float2(0.f, 0.f), a1 = a0;
      const int quads = (cnt + 3) / 4;
#pragma unroll 4
      for (int k = 0; k < quads; k++) {
        const float4 a = ar[k], w = wr[k];
        a0 = __ffma2_rn(make_float2(a.x, a.y), make_float2(w.x, w.y), a0);
        a1 = __ffma2_rn(make_float2(a.z, a.w), make_float2(w.z, w.w), a1);
      }
      if (nn <= p && (mm > 0 || c == 0)) {
        const double f = fac[ifull_d(nn, mm)] * c_monic.g[nn * (nn + 1) / 2 + mm];
        const double v = (c ? -f : f) * (double)((a0.x + a0.y) + (a1.x + a1.y));
        double* o = M + (size_t)b * K + nn * nn + (mm ? 2 * mm - 1 + c : 0);
        if (shared_leaf) atomicAdd(o, v);
        else *o = v;
      }
    }
    __syncwarp();
  };
#pragma unroll
  for (int m = 0; m <= P; m++) {
    if (m > 0) {
      const float2 t = __ffma2_rn(tr, x, __fmul2_rn(ti, ny));
      ti = __ffma2_rn(tr, y, __fmul2_rn(ti, x));
      tr = t;
    }
    if (rows + P + 1 - m > kFRows) {
      flush(rows, m0);
      rows = 0;
    }
    if (rows == 0) m0 = m;
    reinterpret_cast<float2*>(sW[warp][2 * (m - m0)])[lane] = tr;
    reinterpret_cast<float2*>(sW[warp][2 * (m - m0) + 1])[lane] = ti;
    float2 b1 = make_float2(1.f, 1.f), b2 = make_float2(0.f, 0.f);
#pragma unroll
    for (int n = m; n <= P; n++, rows++) {
      reinterpret_cast<float2*>(sA[warp][rows])[lane] = b1;
      if (n < P) {
        const float c = monic_c(n + 1, m);
        const float2 bn = n == m ? __fmul2_rn(z, b1)
                                 : __ffma2_rn(z, b1, __fmul2_rn(__fmul2_rn(make_float2(c, c), mr2), b2));
        b2 = b1;
        b1 = bn;
      }
    }
  }
  flush(rows, m0);
}

// ------------------------------------------------------------------ P2M (FP32)
// Mixed-precision P2M of dipoles: one thread per source point evaluates every S_n^m of
// its point in FP32 with the degree rows held in registers (order P fixed at
// compile time, runtime order p <= P), writes its contributions to shared
// memory, and the block reduces the columns in FP64.  The multipole of a leaf
// carries FP32 rounding of each point's terms (relative 1e-7) -- below the
// tensor-core error of the translations that consume it.  A block is one work
// item of up to kP2MItem sources of a leaf, so that the dense leaves of
// clustered points (a thousand points and more) spread over many SMs; a leaf
// of several items is summed with FP64 atomics into zeroed rows.
__constant__ float c_fac32[21 * 21 + 21];  // fac(n, m) at n*n+n+m, n <= 20

constexpr int kP2MThreads = kP2MItem;

template <int P>
__global__ void __launch_bounds__(kP2MThreads) p2m_f32(int p, int K, const int2* __restrict__ work,
                                                       const int* __restrict__ keys,
                                                       const int2* __restrict__ leaf, const float4* __restrict__ spos,
                                                       const float4* __restrict__ snrm, const float* __restrict__ qs,
                                                       float xmin, float ymin, float zmin, double rb,
                                                       double* __restrict__ M) {
  extern __shared__ float contrib[];  // [kP2MThreads][K]
  const int2 wk = work[blockIdx.x];
  const int b = wk.x;
  double xc, yc, zc;
  box_center(keys[b], xmin, ymin, zmin, rb, xc, yc, zc);
  const int2 leaf_b = leaf[b];
  const bool shared_leaf = leaf_b.y > kP2MThreads;  // summed by several items
  const int2 lf = make_int2(leaf_b.x + wk.y, min(kP2MThreads, leaf_b.y - wk.y));
  const double inv_rb = 1.0 / rb;
  double acc[(P + 1) * (P + 1) / kP2MThreads + 1];
#pragma unroll
  for (int i = 0; i < (P + 1) * (P + 1) / kP2MThreads + 1; i++) acc[i] = 0.0;
  float* my = contrib + threadIdx.x * K;
  for (int j0 = 0; j0 < lf.y; j0 += kP2MThreads) {
    const int jj = j0 + threadIdx.x;
    const bool act = jj < lf.y;
    const int j = lf.x + (act ? jj : 0);
    const float4 xs = spos[j];
    const float q = act ? qs[j] : 0.f;
    const float x = (float)(((double)xs.x - xc) * inv_rb), y = (float)(((double)xs.y - yc) * inv_rb),
                z = (float)(((double)xs.z - zc) * inv_rb);
    const float r2 = x * x + y * y + z * z;
    const float4 nv = snrm[j];
    const float s = q * (float)inv_rb, qnx = s * nv.x, qny = s * nv.y, qnz = s * nv.z;
    float r1re[P + 1], r1im[P + 1], r2re[P + 1], r2im[P + 1];
#pragma unroll
    for (int m = 0; m <= P; m++) r1re[m] = r1im[m] = r2re[m] = r2im[m] = 0.f;
#pragma unroll
    for (int n = 0; n <= P; n++) {
      float cre[P + 1], cim[P + 1];
#pragma unroll
      for (int m = 0; m <= P; m++) {
        cre[m] = cim[m] = 0.f;
        if (m > n) continue;
        if (n == 0) {
          cre[0] = 1.f;
        } else if (m == n) {  // S_n^n = -(2n-1) (x + i y) S_{n-1}^{n-1}
          const float a = -(2.f * n - 1.f);
          cre[m] = a * (x * r1re[n - 1] - y * r1im[n - 1]);
          cim[m] = a * (x * r1im[n - 1] + y * r1re[n - 1]);
        } else if (m == n - 1) {
          const float a = (2.f * n - 1.f) * z;
          cre[m] = a * r1re[m];
          cim[m] = a * r1im[m];
        } else {
          const float inv = 1.f / (float)(n - m);
          const float a = (2.f * n - 1.f) * z * inv, c = (float)(n + m - 1) * r2 * inv;
          cre[m] = a * r1re[m] - c * r2re[m];
          cim[m] = a * r1im[m] - c * r2im[m];
        }
        if (n > p) continue;
        float vre, vim;
        if (n == 0) {
          vre = vim = 0.f;
        } else {
          // n . grad S_n^m from degree n-1
          const float upr = (m + 1 <= n - 1) ? r1re[m + 1 <= P ? m + 1 : P] : 0.f;
          const float upi = (m + 1 <= n - 1) ? r1im[m + 1 <= P ? m + 1 : P] : 0.f;
          float dnr, dni, cm;
          if (m == 0) {  // conj(S_{n-1}^1)
            dnr = (n - 1 >= 1) ? r1re[1 <= P ? 1 : P] : 0.f;
            dni = (n - 1 >= 1) ? -r1im[1 <= P ? 1 : P] : 0.f;
            cm = 1.f;
          } else {
            dnr = r1re[m - 1 >= 0 ? m - 1 : 0];
            dni = r1im[m - 1 >= 0 ? m - 1 : 0];
            cm = -(float)(n + m) * (float)(n + m - 1);
          }
          const float s1r = (m <= n - 1) ? r1re[m] : 0.f, s1i = (m <= n - 1) ? r1im[m] : 0.f;
          // D = 1/2 (nx - i ny) up + 1/2 cm (nx + i ny) dn + nz (n+m) s1
          const float Dre = 0.5f * (qnx * upr + qny * upi) + 0.5f * cm * (qnx * dnr - qny * dni) + qnz * (n + m) * s1r;
          const float Dim = 0.5f * (qnx * upi - qny * upr) + 0.5f * cm * (qnx * dni + qny * dnr) + qnz * (n + m) * s1i;
          const float f = c_fac32[n * n + n + m];
          vre = f * Dre;
          vim = -f * Dim;
        }
        if (m == 0) my[n * n] = vre;
        else {
          my[n * n + 2 * m - 1] = vre;
          my[n * n + 2 * m] = vim;
        }
      }
#pragma unroll
      for (int m = 0; m <= P; m++) {
        r2re[m] = r1re[m];
        r2im[m] = r1im[m];
        r1re[m] = cre[m];
        r1im[m] = cim[m];
      }
    }
    __syncthreads();
    // column sums over the chunk's points (inactive points contributed zeros)
#pragma unroll
    for (int i = 0; i < (P + 1) * (P + 1) / kP2MThreads + 1; i++) {
      const int k = threadIdx.x + i * kP2MThreads;
      if (k < K) {
        float t = 0.f;
        const int npt = min(kP2MThreads, lf.y - j0);
        for (int pt = 0; pt < npt; pt++) t += contrib[pt * K + k];
        acc[i] += (double)t;
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < (P + 1) * (P + 1) / kP2MThreads + 1; i++) {
    const int k = threadIdx.x + i * kP2MThreads;
    if (k < K) {
      if (shared_leaf) atomicAdd(M + (size_t)b * K + k, acc[i]);
      else M[(size_t)b * K + k] = acc[i];
    }
  }
}

// ------------------------------------------------------------------ L2P
// One block (64 threads) per work item of up to 128 targets of a leaf, two
// targets a thread.  The leaf's local expansion is turned once into the
// coefficients of the potential (C_F) and of its three derivatives by the
// ladder identities above (C_z; the x and y derivatives as the real part of
// C_X S and the imaginary part of C_Y S); with S_n^m = A_n^m s_m, A real, a thread
// sums the coefficients of an order over its degrees as reals times A and
// multiplies by the complex s_m once per order.
// Bound: the FP64 pipe and the recurrence's latency.  (One block per leaf and
// complex sums per term: 262,144 clustered points, p = 12: 0.37 ms; 0.07 now.
// The same loops in FP32, two targets side by side, ran the mixed form's L2P of
// 1,048,576 points in 0.25 ms against 0.20 of the unrolled l2p_f32.)
constexpr int kL2PThreads = 64;

// POT / DER: the potential, its derivatives
template <int KER, bool POT, bool DER>
__global__ void __launch_bounds__(kL2PThreads) l2p_cart(int p, int K, const int2* __restrict__ work,
                                                   const int* __restrict__ keys, const int2* __restrict__ leaf,
                                                   const float4* __restrict__ tpos, const float4* __restrict__ tnrm,
                                                   const double* __restrict__ fac, float xmin, float ymin, float zmin,
                                                   double rb, double coef, const double* __restrict__ L,
                                                   double* __restrict__ pot, double* __restrict__ grad, int ni) {
  constexpr int NS = (POT ? 1 : 0) + (DER ? 3 : 0);  // complex sums per order
  extern __shared__ double2 C[];                     // their coefficients [terms, by order][NS]
  const int NT = (p + 1) * (p + 2) / 2;
  const int2 wk = work[blockIdx.x];
  const int b = wk.x;
  const double* Lb = L + (size_t)b * K;
  auto Lnm = [&](int n, int m) -> cplx {
    if (m == 0) return {Lb[n * n], 0.0};
    return {Lb[n * n + 2 * m - 1], Lb[n * n + 2 * m]};
  };
  for (int idx = threadIdx.x; idx < NT; idx += kL2PThreads) {
    int n = 0;
    while ((n + 1) * (n + 2) / 2 <= idx) n++;
    const int m = idx - n * (n + 1) / 2;
    const double wm = m ? 2.0 : 1.0;
    double2* c = C + NS * (m * (p + 1) - m * (m - 1) / 2 + n - m);
    auto put = [&](int k, cplx v) { c[k] = make_double2(v.re, v.im); };
    if (POT) put(0, cscale(Lnm(n, m), wm * fac[ifull_d(n, m)]));
    if (DER) {
      cplx cz = {0.0, 0.0}, cx = cz, cy = cz;
      if (n < p) {
        cz = cscale(Lnm(n + 1, m), wm * fac[ifull_d(n + 1, m)] * (n + 1 + m));
        const cplx cp = m >= 1 ? cscale(Lnm(n + 1, m - 1), (m - 1 ? 2.0 : 1.0) * fac[ifull_d(n + 1, m - 1)]) : cplx{0.0, 0.0};
        const cplx cm = cscale(Lnm(n + 1, m + 1), -2.0 * fac[ifull_d(n + 1, m + 1)] * (double)(n + m + 2) * (double)(n + m + 1));
        const double cs = m == 1 ? fac[ifull_d(n + 1, 0)] * Lb[(n + 1) * (n + 1)] : 0.0;  // of conj(S_n^1)
        cx = {cp.re + cm.re + cs, cp.im + cm.im};
        cy = {cp.re - cm.re + cs, cp.im - cm.im};
      }
      put(NS - 3, cz);
      put(NS - 2, cx);
      put(NS - 1, cy);
    }
  }
  __syncthreads();
  double xc, yc, zc;
  box_center(keys[b], xmin, ymin, zmin, rb, xc, yc, zc);
  const int2 lf = leaf[b];
  const double inv_rb = 1.0 / rb;
  const int i0 = wk.y + threadIdx.x, end = min(lf.y, wk.y + 2 * kL2PThreads);
  if (i0 >= end) return;
  const int it[2] = {lf.x + i0, lf.x + (i0 + kL2PThreads < end ? i0 + kL2PThreads : i0)};
  double x[2], y[2], z[2], r2[2], sr[2], si[2];
  double F[2] = {0, 0}, gx[2] = {0, 0}, gy[2] = {0, 0}, gz[2] = {0, 0};
#pragma unroll
  for (int t = 0; t < 2; t++) {
    const float4 v = tpos[it[t]];
    x[t] = ((double)v.x - xc) * inv_rb;
    y[t] = ((double)v.y - yc) * inv_rb;
    z[t] = ((double)v.z - zc) * inv_rb;
    r2[t] = x[t] * x[t] + y[t] * y[t] + z[t] * z[t];
    sr[t] = 1.0;
    si[t] = 0.0;
  }
  const double2* c = C;
  for (int m = 0; m <= p; m++) {
    double ur[2][NS], ui[2][NS], a1[2], a2[2];  // sums; A_n^m, A_{n-1}^m
#pragma unroll
    for (int t = 0; t < 2; t++) {
      if (m > 0) {  // s_m = -(2m-1) (x + i y) s_{m-1}
        const double f = -(2.0 * m - 1.0), tr = f * (sr[t] * x[t] - si[t] * y[t]);
        si[t] = f * (sr[t] * y[t] + si[t] * x[t]);
        sr[t] = tr;
      }
      a1[t] = 1.0;
      a2[t] = 0.0;
#pragma unroll
      for (int k = 0; k < NS; k++) ur[t][k] = ui[t][k] = 0.0;
    }
    for (int n = m;; n++) {
#pragma unroll
      for (int k = 0; k < NS; k++) {
        const double2 ck = c[k];
#pragma unroll
        for (int t = 0; t < 2; t++) {
          ur[t][k] = fma(ck.x, a1[t], ur[t][k]);
          ui[t][k] = fma(ck.y, a1[t], ui[t][k]);
        }
      }
      c += NS;
      if (n == p) break;
      const double2 ab = c_rec[(n + 1) * (n + 2) / 2 + m];
#pragma unroll
      for (int t = 0; t < 2; t++) {
        const double an = fma(ab.x * z[t], a1[t], -(ab.y * r2[t]) * a2[t]);
        a2[t] = a1[t];
        a1[t] = an;
      }
    }
    // times s_m: the potential and d/dz the real parts, d/dx the real part of X s, d/dy the imaginary part of Y s
#pragma unroll
    for (int t = 0; t < 2; t++) {
      if (POT) F[t] += ur[t][0] * sr[t] - ui[t][0] * si[t];
      if (DER) {
        gz[t] += ur[t][NS - 3] * sr[t] - ui[t][NS - 3] * si[t];
        gx[t] += ur[t][NS - 2] * sr[t] - ui[t][NS - 2] * si[t];
        gy[t] += ur[t][NS - 1] * si[t] + ui[t][NS - 1] * sr[t];
      }
    }
  }
  const double c1 = coef * inv_rb, c2 = coef * inv_rb * inv_rb;
#pragma unroll
  for (int t = 0; t < 2; t++) {
    if (t == 1 && i0 + kL2PThreads >= end) break;
    const int i = it[t];
    if (KER == FMMB_LAPLACE_GNI) {
      const float4 nv = tnrm[i];
      pot[i] = -c2 * ((double)nv.x * (0.5 * gx[t]) + (double)nv.y * (0.5 * gy[t]) + (double)nv.z * gz[t]);
    } else {
      pot[i] = c1 * F[t];
      if (DER) {  // G and Gnj: the local expansion is the potential itself
        grad[i] = c2 * (0.5 * gx[t]);
        grad[ni + (size_t)i] = c2 * (0.5 * gy[t]);
        grad[2 * (size_t)ni + i] = c2 * gz[t];
      }
    }
  }
}

// ------------------------------------------------------------------ L2P, Hessian
// The gradient w.r.t. the target position of the far-field Gni potential
// -(1/4pi) n . grad(phi) (normal held fixed): -(1/4pi) H n, H the Hessian of
// the local expansion.  One block (64 threads) per target leaf.  With F the
// real potential of L in scaled coordinates written over all orders,
// F = sum_{n, |m| <= n} b_n^m S_n^m (b_n^m = fac(n,m) L_n^m for m >= 0,
// b_n^{-m} = (-1)^m (n+m)!/(n-m)! conj(b_n^m)), the ladder identities give its
// derivatives as expansions of one degree less:
//   d/dx F: c_{n-1}^k = (b_n^{k-1} - (n+k+1)(n+k) b_n^{k+1}) / 2
//   d/dy F: c_{n-1}^k = (b_n^{k-1} + (n+k+1)(n+k) b_n^{k+1}) / (2i)
//   d/dz F: c_{n-1}^k = (n+k) b_n^k
// i.e. local expansions L^D = c / fac of the same form (real potentials); the
// gradient of each, evaluated like l2p_cart's, is one row of H.
constexpr int kL2PHThreads = 64;

__global__ void __launch_bounds__(kL2PHThreads) l2p_hess_gni(int p, int K, const int* __restrict__ keys,
                                                             const int2* __restrict__ leaf,
                                                             const float4* __restrict__ tpos,
                                                             const float4* __restrict__ tnrm,
                                                             const double* __restrict__ fac, float xmin, float ymin,
                                                             float zmin, double rb, double coef,
                                                             const double* __restrict__ L, double* __restrict__ grad,
                                                             int ni) {
  extern __shared__ double sm[];
  const int P = (p + 1) * (p + 2) / 2;
  cplx* Ld = reinterpret_cast<cplx*>(sm);  // [3][P] derivative expansions (m >= 0)
  cplx* Cz = Ld + 3 * P;                   // [3][P] their gradient coefficient sets
  cplx* Cp = Cz + 3 * P;
  cplx* Cm = Cp + 3 * P;
  double* Cs = reinterpret_cast<double*>(Cm + 3 * P);  // [3][p+1]
  const int b = blockIdx.x;
  const double* Lb = L + (size_t)b * K;
  auto bnm = [&](int n, int m) -> cplx {  // b_n^m for -1 <= m
    if (n < 0 || m > n || n > p) return {0.0, 0.0};
    if (m == -1) {
      if (n < 1) return {0.0, 0.0};
      const double f = fac[ifull_d(n, 1)];
      return {-(double)n * (n + 1) * f * Lb[n * n + 1], (double)n * (n + 1) * f * Lb[n * n + 2]};
    }
    if (m == 0) return {fac[ifull_d(n, 0)] * Lb[n * n], 0.0};
    const double f = fac[ifull_d(n, m)];
    return {f * Lb[n * n + 2 * m - 1], f * Lb[n * n + 2 * m]};
  };
  for (int idx = threadIdx.x; idx < P; idx += blockDim.x) {
    int n1 = 0;
    while ((n1 + 1) * (n1 + 2) / 2 <= idx) n1++;
    const int k = idx - n1 * (n1 + 1) / 2;  // degree n1 = n - 1, order k
    cplx cx = {0.0, 0.0}, cy = {0.0, 0.0}, cz = {0.0, 0.0};
    if (n1 < p) {
      const int n = n1 + 1;
      const cplx lo = bnm(n, k - 1), hi = bnm(n, k + 1), mid = bnm(n, k);
      const double a = (double)(n + k + 1) * (double)(n + k);
      cx = {0.5 * (lo.re - a * hi.re), 0.5 * (lo.im - a * hi.im)};
      const cplx t = {lo.re + a * hi.re, lo.im + a * hi.im};
      cy = {0.5 * t.im, -0.5 * t.re};  // t / (2i)
      cz = {(n + k) * mid.re, (n + k) * mid.im};
    }
    const double inv = 1.0 / fac[ifull_d(n1, k)];
    Ld[idx] = cscale(cx, inv);
    Ld[P + idx] = cscale(cy, inv);
    Ld[2 * P + idx] = cscale(cz, inv);
    if (k == 0) {  // real by construction; drop the rounding residue
      Ld[idx].im = Ld[P + idx].im = Ld[2 * P + idx].im = 0.0;
    }
  }
  __syncthreads();
  // gradient coefficient sets of each derivative expansion (as l2p_cart's of L)
  for (int e = threadIdx.x; e < 3 * P; e += blockDim.x) {
    const int d = e / P, idx = e % P;
    const cplx* Lx = Ld + d * P;
    auto Lnm = [&](int n, int m) -> cplx { return Lx[n * (n + 1) / 2 + m]; };
    int n = 0;
    while ((n + 1) * (n + 2) / 2 <= idx) n++;
    const int m = idx - n * (n + 1) / 2;
    const double wm = m ? 2.0 : 1.0;
    if (n < p) {
      Cz[e] = cscale(Lnm(n + 1, m), wm * fac[ifull_d(n + 1, m)] * (n + 1 + m));
      Cp[e] = (m >= 1) ? cscale(Lnm(n + 1, m - 1), (m - 1 ? 2.0 : 1.0) * fac[ifull_d(n + 1, m - 1)]) : cplx{0.0, 0.0};
      Cm[e] = (m + 1 <= n + 1) ? cscale(Lnm(n + 1, m + 1), -2.0 * fac[ifull_d(n + 1, m + 1)] * (double)(n + m + 2) *
                                                                (double)(n + m + 1))
                               : cplx{0.0, 0.0};
    } else {
      Cz[e] = Cp[e] = Cm[e] = cplx{0.0, 0.0};
    }
  }
  for (int e = threadIdx.x; e < 3 * (p + 1); e += blockDim.x) {
    const int d = e / (p + 1), n = e % (p + 1);
    Cs[e] = (n < p) ? fac[ifull_d(n + 1, 0)] * Ld[d * P + (n + 1) * (n + 2) / 2].re : 0.0;
  }
  __syncthreads();
  double xc, yc, zc;
  box_center(keys[b], xmin, ymin, zmin, rb, xc, yc, zc);
  const int2 lf = leaf[b];
  const double inv_rb = 1.0 / rb;
  for (int ii = threadIdx.x; ii < lf.y; ii += blockDim.x) {
    const int i = lf.x + ii;
    const float4 xt = tpos[i];
    const double x = ((double)xt.x - xc) * inv_rb, y = ((double)xt.y - yc) * inv_rb, z = ((double)xt.z - zc) * inv_rb;
    const double r2 = x * x + y * y + z * z;
    double dzr[3] = {0, 0, 0}, dpr[3] = {0, 0, 0}, dpi[3] = {0, 0, 0}, dmr[3] = {0, 0, 0}, dmi[3] = {0, 0, 0};
    cplx smm = {1.0, 0.0};
    for (int m = 0; m <= p; m++) {
      if (m > 0) smm = cscale(cmul(smm, cplx{x, y}), -(2.0 * m - 1.0));
      cplx s1 = {0.0, 0.0}, s2 = {0.0, 0.0};
      for (int n = m; n < p; n++) {  // the derivative expansions stop at degree p - 1
        cplx sn;
        if (n == m) sn = smm;
        else if (n == m + 1) sn = cscale(s1, (2.0 * m + 1.0) * z);
        else {
          const double inv = c_inv[n - m];
          const double a = (2.0 * n - 1.0) * z * inv, c = (n + m - 1.0) * r2 * inv;
          sn = {a * s1.re - c * s2.re, a * s1.im - c * s2.im};
        }
        const int idx = n * (n + 1) / 2 + m;
#pragma unroll
        for (int d = 0; d < 3; d++) {
          const cplx cz = Cz[d * P + idx], cp = Cp[d * P + idx], cmm = Cm[d * P + idx];
          dzr[d] += cz.re * sn.re - cz.im * sn.im;
          dpr[d] += cp.re * sn.re - cp.im * sn.im;
          dpi[d] += cp.re * sn.im + cp.im * sn.re;
          dmr[d] += cmm.re * sn.re - cmm.im * sn.im;
          dmi[d] += cmm.re * sn.im + cmm.im * sn.re;
          if (m == 1) {
            dmr[d] += Cs[d * (p + 1) + n] * sn.re;
            dmi[d] -= Cs[d * (p + 1) + n] * sn.im;
          }
        }
        s2 = s1;
        s1 = sn;
      }
    }
    const float4 nv = tnrm[i];
    const double nn[3] = {(double)nv.x, (double)nv.y, (double)nv.z};
    double hn[3] = {0, 0, 0};  // H n in scaled coordinates (H symmetric: row d of H is grad(d/dd F))
#pragma unroll
    for (int d = 0; d < 3; d++) {
      hn[0] += nn[d] * 0.5 * (dpr[d] + dmr[d]);
      hn[1] += nn[d] * 0.5 * (dpi[d] - dmi[d]);
      hn[2] += nn[d] * dzr[d];
    }
    const double c3 = -coef * inv_rb * inv_rb * inv_rb;
    grad[i] = c3 * hn[0];
    grad[ni + i] = c3 * hn[1];
    grad[2 * ni + i] = c3 * hn[2];
  }
}

// FP32 L2P for the mixed form, one thread per target, one block per work item of
// up to 128 targets of a leaf.  As l2p_cart, S_n^m = A_n^m s_m: the coefficients of
// an order are summed over its degrees as reals times A and multiplied by the
// complex s_m once per order; here in the monic form (c_monic, above), fully
// unrolled to order P (runtime order p <= P).  Coefficients are formed in
// FP64 and rounded; B, the powers of t and the sums of one order are FP32, the
// sums over the orders and the terms of degree 0 of the potential and of each
// derivative, the largest, FP64 (in the FP32 sums those made the gradient's
// rounding error 7e-8 of it, 1e-8 to 2.3e-8 now).
// Bound: the FP32 pipe: 3 + 8 lane operations a term and two 16-byte
// shared-memory reads.  (Complex recurrences and derivative sums per term, 16
// operations and three reads: 1,048,576 targets at p = 12: 0.20 ms; 0.11 now.)
constexpr int kL2PF32Threads = 128;

// POT / DER: the potential, its derivatives
template <int KER, bool POT, bool DER, int P>
__global__ void __launch_bounds__(kL2PF32Threads) l2p_f32(int p, int K, const int2* __restrict__ work,
                                                          const int* __restrict__ keys,
                                                          const int2* __restrict__ leaf, const float4* __restrict__ tpos,
                                                          const float4* __restrict__ tnrm, const double* __restrict__ fac,
                                                          float xmin, float ymin, float zmin, double rb, double coef,
                                                          const double* __restrict__ L, double* __restrict__ pot,
                                                          double* __restrict__ grad, int ni) {
  constexpr int NT = (P + 1) * (P + 2) / 2;
  __shared__ float4 CA[DER ? NT : 1], CB[DER ? NT : 1];  // (d/dx, d/dy), (d/dz, potential), by order
  __shared__ float2 CF[DER ? 1 : NT];                    // the potential alone
  const int2 wk = work[blockIdx.x];
  const int b = wk.x;
  const double* Lb = L + (size_t)b * K;
  auto Lnm = [&](int n, int m) -> cplx {
    if (m == 0) return {Lb[n * n], 0.0};
    return {Lb[n * n + 2 * m - 1], Lb[n * n + 2 * m]};
  };
  auto f2 = [](cplx c) { return make_float2((float)c.re, (float)c.im); };
  for (int idx = threadIdx.x; idx < NT; idx += kL2PF32Threads) {
    int n = 0;
    while ((n + 1) * (n + 2) / 2 <= idx) n++;
    const int m = idx - n * (n + 1) / 2;
    const int at = m * (P + 1) - m * (m - 1) / 2 + n - m;
    const double g = c_monic.g[idx], wm = m ? 2.0 : 1.0;
    float2 cf = make_float2(0.f, 0.f), cx = cf, cy = cf, cz = cf;
    if (n > 0 && n <= p && POT) cf = f2(cscale(Lnm(n, m), g * wm * fac[ifull_d(n, m)]));
    if (DER && n > 0 && n < p) {  // as l2p_cart
      cz = f2(cscale(Lnm(n + 1, m), g * wm * fac[ifull_d(n + 1, m)] * (n + 1 + m)));
      const cplx cp = m >= 1 ? cscale(Lnm(n + 1, m - 1), (m - 1 ? 2.0 : 1.0) * fac[ifull_d(n + 1, m - 1)]) : cplx{0.0, 0.0};
      const cplx cm = cscale(Lnm(n + 1, m + 1), -2.0 * fac[ifull_d(n + 1, m + 1)] * (double)(n + m + 2) * (double)(n + m + 1));
      const double cs = m == 1 ? fac[ifull_d(n + 1, 0)] * Lb[(n + 1) * (n + 1)] : 0.0;
      cx = f2({g * (cp.re + cm.re + cs), g * (cp.im + cm.im)});
      cy = f2({g * (cp.re - cm.re + cs), g * (cp.im - cm.im)});
    }
    if (DER) {
      CA[at] = make_float4(cx.x, cx.y, cy.x, cy.y);
      CB[at] = make_float4(cz.x, cz.y, cf.x, cf.y);
    } else {
      CF[at] = cf;
    }
  }
  __syncthreads();
  double xc, yc, zc;
  box_center(keys[b], xmin, ymin, zmin, rb, xc, yc, zc);
  const int2 lf = leaf[b];
  const double inv_rb = 1.0 / rb;
  const int it = wk.y + threadIdx.x;
  if (it >= lf.y) return;
  const int i = lf.x + it;
  const float4 xt = tpos[i];
  const float x = (float)(((double)xt.x - xc) * inv_rb), y = (float)(((double)xt.y - yc) * inv_rb),
              z = (float)(((double)xt.z - zc) * inv_rb);
  const float mr2 = -(x * x + y * y + z * z);
  double F = 0, gx = 0, gy = 0, gz = 0;
  if (POT) F = Lb[0] * fac[0];
  if (DER) {  // p >= 1: d/dz from (1, 0), d/dx and d/dy (twice) from (1, 1)
    const double f11 = 4.0 * fac[ifull_d(1, 1)];
    gx = -f11 * Lb[2];
    gy = f11 * Lb[3];
    gz = fac[ifull_d(1, 0)] * Lb[1];
  }
  float tr = 1.f, ti = 0.f;  // t^m
#pragma unroll
  for (int m = 0; m <= P; m++) {
    if (m > 0) {
      const float t = tr * x - ti * y;
      ti = tr * y + ti * x;
      tr = t;
    }
    const float2 zero = make_float2(0.f, 0.f);
    float2 uf = zero, ux = zero, uy = zero, uz = zero;
    float b1 = 1.f, b2 = 0.f;
#pragma unroll
    for (int n = m; n <= P; n++) {
      const int at = m * (P + 1) - m * (m - 1) / 2 + n - m;
      const float2 bb = make_float2(b1, b1);
      if (DER) {
        const float4 ca = CA[at], cb = CB[at];
        ux = __ffma2_rn(make_float2(ca.x, ca.y), bb, ux);
        uy = __ffma2_rn(make_float2(ca.z, ca.w), bb, uy);
        uz = __ffma2_rn(make_float2(cb.x, cb.y), bb, uz);
        if (POT) uf = __ffma2_rn(make_float2(cb.z, cb.w), bb, uf);
      } else {
        uf = __ffma2_rn(CF[at], bb, uf);
      }
      if (n < P) {
        const float bn = n == m ? z * b1 : fmaf(z, b1, (monic_c(n + 1, m) * mr2) * b2);
        b2 = b1;
        b1 = bn;
      }
    }
    // times t^m: potential and d/dz the real parts, d/dx the real part of X s, d/dy the imaginary part of Y s
    if (POT) F += (double)(uf.x * tr - uf.y * ti);
    if (DER) {
      gx += (double)(ux.x * tr - ux.y * ti);
      gy += (double)(uy.x * ti + uy.y * tr);
      gz += (double)(uz.x * tr - uz.y * ti);
    }
  }
  const double c1 = coef * inv_rb, c2 = coef * inv_rb * inv_rb;
  if (KER == FMMB_LAPLACE_GNI) {
    const float4 nv = tnrm[i];
    pot[i] = -c2 * ((double)nv.x * (0.5 * gx) + (double)nv.y * (0.5 * gy) + (double)nv.z * gz);
  } else {
    pot[i] = c1 * F;
    if (DER) {
      grad[i] = c2 * (0.5 * gx);
      grad[ni + (size_t)i] = c2 * (0.5 * gy);
      grad[2 * (size_t)ni + i] = c2 * gz;
    }
  }
}

template <int P>
void l2p_f32_launch(int kernel, int nwork, const int2* work, int p, int K, const int* keys, const int2* leaf,
                    const float4* tpos, const float4* tnrm, const double* fac, const float* bbox, double rb,
                    double coef, const double* L, double* pot, double* grad, int ni, cudaStream_t st) {
  auto go = [&](auto k) {
    k<<<nwork, kL2PF32Threads, 0, st>>>(p, K, work, keys, leaf, tpos, tnrm, fac, bbox[0], bbox[1], bbox[2], rb, coef, L,
                                        pot, grad, ni);
  };
  if (kernel == FMMB_LAPLACE_GNI) go(l2p_f32<FMMB_LAPLACE_GNI, false, true, P>);
  else if (kernel == FMMB_LAPLACE_G && grad) go(l2p_f32<FMMB_LAPLACE_G, true, true, P>);
  else go(l2p_f32<FMMB_LAPLACE_G, true, false, P>);
}

}  // namespace

void launch_p2m_dmma(int kernel, int nleaf, int p, int K, const int* keys, const int2* leaf, const float4* spos,
                    const float4* snrm, const float* qs, const double* fac, const Sem& s, const float* bbox, double rb,
                    double* M, cudaStream_t st) {
  if (nleaf <= 0) return;
  const bool dip = kernel == FMMB_LAPLACE_GNJ;
  const int ncol = dip ? 6 : 2;
  const size_t sm = ((size_t)ncol * (p + 1) * (p + 2) / 2 + (kPts / 32) * (size_t)(kRows + ncol) * kPS) * sizeof(double);
  auto go = [&](auto k) {
    k<<<nleaf, kPts, sm, st>>>(p, K, keys, leaf, spos, snrm, qs, fac, s, bbox[0], bbox[1], bbox[2], rb, M);
  };
  if (dip) go(p2m_dmma<FMMB_LAPLACE_GNJ, false>);
  else if (s.ref) go(p2m_dmma<FMMB_LAPLACE_G, true>);
  else go(p2m_dmma<FMMB_LAPLACE_G, false>);
  FMMB_CHECK_LAUNCH();
}

namespace {
template <int P>
void p2m_f32_launch(int kernel, int nwork, const int2* work, int p, int K, const int* keys, const int2* leaf,
                    const float4* spos, const float4* snrm, const float* qs, const double* fac, const float* bbox, double rb,
                    double* M, cudaStream_t st) {
  const size_t sm = (size_t)kP2MThreads * K * sizeof(float);
  if (kernel == FMMB_LAPLACE_GNJ)
    p2m_f32<P><<<nwork, kP2MThreads, sm, st>>>(p, K, work, keys, leaf, spos, snrm, qs, bbox[0], bbox[1], bbox[2], rb, M);
  else
    p2m_f32_charges<P><<<(nwork + kFWarps - 1) / kFWarps, 32 * kFWarps, 0, st>>>(
        p, K, nwork, work, keys, leaf, spos, qs, fac, bbox[0], bbox[1], bbox[2], rb, M);
}
}  // namespace

void init_fac32() {
  static bool done[64] = {};
  int dev = 0;
  FMMB_CUDA(cudaGetDevice(&dev));
  if (dev < 64 && done[dev]) return;
  float h[21 * 21 + 21] = {};
  for (int n = 0; n <= 20; n++)
    for (int m = 0; m <= n; m++) {
      double f = 1.0;  // sqrt((n-m)!/(n+m)!)
      for (int k = n - m + 1; k <= n + m; k++) f /= k;
      h[n * n + n + m] = (float)std::sqrt(f);
    }
  FMMB_CUDA(cudaMemcpyToSymbol(c_fac32, h, sizeof(h)));
  if (dev < 64) done[dev] = true;
}

bool launch_p2m_f32(int kernel, int nwork, const int2* work, int p, int K, const int* keys, const int2* leaf,
                    const float4* spos, const float4* snrm, const float* qs, const double* fac, const float* bbox,
                    double rb, double* M, cudaStream_t st) {
  if (p > 12) return false;  // FP64 above
  if (nwork <= 0) return true;
  if (p <= 8) p2m_f32_launch<8>(kernel, nwork, work, p, K, keys, leaf, spos, snrm, qs, fac, bbox, rb, M, st);
  else if (p <= 10) p2m_f32_launch<10>(kernel, nwork, work, p, K, keys, leaf, spos, snrm, qs, fac, bbox, rb, M, st);
  else p2m_f32_launch<12>(kernel, nwork, work, p, K, keys, leaf, spos, snrm, qs, fac, bbox, rb, M, st);
  FMMB_CHECK_LAUNCH();
  return true;
}

void launch_l2p_cart(int kernel, int nwork, const int2* work, int p, int K, const int* keys, const int2* leaf,
                     const float4* tpos, const float4* tnrm, const double* fac, const float* bbox, double rb, double coef,
                     const double* L, double* pot, double* grad, int ni, cudaStream_t st) {
  if (nwork <= 0) return;
  const size_t terms = (size_t)(p + 1) * (p + 2) / 2;
  auto go = [&](auto k, int ns) {
    k<<<nwork, kL2PThreads, terms * ns * sizeof(double2), st>>>(p, K, work, keys, leaf, tpos, tnrm, fac, bbox[0], bbox[1],
                                                                bbox[2], rb, coef, L, pot, grad, ni);
  };
  if (kernel == FMMB_LAPLACE_GNI) go(l2p_cart<FMMB_LAPLACE_GNI, false, true>, 3);
  else if (grad) go(l2p_cart<FMMB_LAPLACE_G, true, true>, 4);
  else go(l2p_cart<FMMB_LAPLACE_G, true, false>, 1);
  FMMB_CHECK_LAUNCH();
}

void launch_l2p_hess_gni(int nleaf, int p, int K, const int* keys, const int2* leaf, const float4* tpos,
                         const float4* tnrm, const double* fac, const float* bbox, double rb, double coef,
                         const double* L, double* grad, int ni, cudaStream_t st) {
  if (nleaf <= 0) return;
  const int P = (p + 1) * (p + 2) / 2;
  const size_t sm = (size_t)12 * P * sizeof(cplx) + 3 * (p + 1) * sizeof(double);
  l2p_hess_gni<<<nleaf, kL2PHThreads, sm, st>>>(p, K, keys, leaf, tpos, tnrm, fac, bbox[0], bbox[1], bbox[2], rb, coef,
                                                L, grad, ni);
  FMMB_CHECK_LAUNCH();
}

bool launch_l2p_f32(int kernel, int nwork, const int2* work, int p, int K, const int* keys, const int2* leaf,
                    const float4* tpos, const float4* tnrm, const double* fac, const float* bbox, double rb,
                    double coef, const double* L, double* pot, double* grad, int ni, cudaStream_t st) {
  if (p > 16) return false;
  if (nwork <= 0) return true;
  if (p <= 8) l2p_f32_launch<8>(kernel, nwork, work, p, K, keys, leaf, tpos, tnrm, fac, bbox, rb, coef, L, pot, grad, ni, st);
  else if (p <= 10) l2p_f32_launch<10>(kernel, nwork, work, p, K, keys, leaf, tpos, tnrm, fac, bbox, rb, coef, L, pot, grad, ni, st);
  else if (p <= 12) l2p_f32_launch<12>(kernel, nwork, work, p, K, keys, leaf, tpos, tnrm, fac, bbox, rb, coef, L, pot, grad, ni, st);
  else l2p_f32_launch<16>(kernel, nwork, work, p, K, keys, leaf, tpos, tnrm, fac, bbox, rb, coef, L, pot, grad, ni, st);
  FMMB_CHECK_LAUNCH();
  return true;
}

}  // namespace fmmb
