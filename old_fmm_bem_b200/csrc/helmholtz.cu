// Complex Helmholtz kernel e^{ikr} / (4 pi r) (FMMB_HELMHOLTZ_G).
//
// The reference's "Helmholtz" is the Yukawa kernel (kernel/Helmholtz_*.cxx);
// the oscillatory kernel has no counterpart there, so this family is written
// from the mathematics:
//
//   e^{ik|x-y|} / (4 pi |x-y|) = ik sum_n j_n(k|y|) h_n(k|x|) sum_m Y_n^m(x^) conj(Y_n^m(y^)),  |x| > |y|
//
// with h_n = j_n + i y_n the spherical Hankel function of the first kind and
// Y_n^m = Ybar_n^|m|(cos t) e^{i m p} the orthonormal spherical harmonics
// (no Condon-Shortley phase; Ybar by the standard fully normalised
// three-term recurrence).  Expansions hold K = (p+1)^2 complex coefficients
// per box, index n^2 + n + m, stored as [re(K) | im(K)]:
//   multipole  phi(x) = sum M_n^m h_n(k r) Y_n^m,  M_n^m = ik sum_j q_j j_n(k rho_j) conj(Y_n^m)
//   local      phi(x) = sum L_n^m j_n(k r) Y_n^m
// Spherical Bessel functions: j_n by Miller's backward recurrence (upward
// when x > n, the power series near 0), y_n by the upward recurrence -- the
// standard methods (e.g. Abramowitz & Stegun 10.1.19, Press et al. 6.7).
//
// Translations (M2M, M2L, L2L) are dense complex K x K operators per level
// and relative position, built here on the GPU by projection: the field of
// one source basis function is sampled on a sphere around the target centre
// (Gauss-Legendre nodes in cos(theta) x equispaced in phi, 2p+8 x 4p+16
// points) and projected on the target basis, conj(Y) and a division by the
// target radial function at the sphere's radius.  The operators are stored in
// the real 2K x 2K form acting on [re | im] (transposed, row stride 2K) and
// applied by the FP64 pair kernel of kernels_fp64.cu; the M2L operators, only
// those at azimuth 0, as the reflection blocks of m2l_parity.cuh.
//
// The same code serves the Yukawa kernel (FMMB_YUKAWA, the reference's neq 10,
// kernel/Helmholtz_G_p2p.cxx:18-23: (pi/2) e^{-lambda r} / (lambda r)) through
//   e^{-l|x-y|} / (4 pi |x-y|) = (2l/pi) sum_n i_n(l|y|) k_n(l|x|) sum_m Y_n^m(x^) conj(Y_n^m(y^))
// with the modified spherical Bessel functions i_n (Miller's backward
// recurrence normalised by i_0 = sinh(x)/x) and k_n (k_0 = (pi/2) e^{-x}/x,
// upward recurrence): real radial functions in place of j_n and h_n, the
// factor 2l/pi in place of ik; the result is scaled by 2 pi^2 / l on output.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "internal.h"
#include "kernels.h"

namespace fmmb {
namespace {

constexpr int kMaxP = 20;

// j_n(x), n = 0..nmax, x >= 0, at j[n ST]
template <int ST = 1>
__device__ void sph_j(int nmax, double x, double* j) {
  if (x < 1e-6) {  // x^n / (2n+1)!! (1 - x^2 / (2 (2n+3)))
    double t = 1.0;
    for (int n = 0; n <= nmax; n++) {
      j[n * ST] = t * (1.0 - x * x / (2.0 * (2 * n + 3)));
      t *= x / (2 * n + 3);
    }
    return;
  }
  double s, c;
  sincos(x, &s, &c);
  const double xi = 1.0 / x, j0 = s * xi, j1 = (j0 - c) * xi;
  j[0] = j0;
  if (nmax == 0) return;
  if (x > (double)nmax) {  // upward recurrence is stable
    j[ST] = j1;
    for (int n = 1; n < nmax; n++) j[(n + 1) * ST] = (2 * n + 1) * xi * j[n * ST] - j[(n - 1) * ST];
    return;
  }
  // Miller: backward from N with arbitrary start, rescaled on the way, then
  // normalised by the larger of j0, j1
  const int N = nmax + 24 + (int)x;
  double jp1 = 0.0, jn = 1e-250;
  for (int n = N; n >= 1; n--) {
    const double jm1 = (2 * n + 1) * xi * jn - jp1;
    jp1 = jn;
    jn = jm1;
    if (n - 1 <= nmax) j[(n - 1) * ST] = jm1;
    if (fabs(jn) > 1e250) {
      jn *= 1e-250;
      jp1 *= 1e-250;
      for (int k = max(n - 1, 0); k <= nmax; k++) j[k * ST] *= 1e-250;
    }
  }
  const double sc = fabs(j0) >= fabs(j1) ? j0 / j[0] : j1 / j[ST];
  for (int n = 0; n <= nmax; n++) j[n * ST] *= sc;
}

// y_n(x), n = 0..nmax, x > 0 (upward recurrence)
__device__ void sph_y(int nmax, double x, double* y) {
  double s, c;
  sincos(x, &s, &c);
  y[0] = -c / x;
  if (nmax >= 1) y[1] = -c / (x * x) - s / x;
  for (int n = 1; n < nmax; n++) y[n + 1] = (2 * n + 1) / x * y[n] - y[n - 1];
}

// i_n(x), n = 0..nmax, x >= 0: Miller's backward recurrence
// i_{n-1} = i_{n+1} + (2n+1)/x i_n, normalised by i_0 = sinh(x)/x
template <int ST = 1>
__device__ void sph_i(int nmax, double x, double* v) {
  if (x < 1e-6) {  // x^n / (2n+1)!! (1 + x^2 / (2 (2n+3)))
    double t = 1.0;
    for (int n = 0; n <= nmax; n++) {
      v[n * ST] = t * (1.0 + x * x / (2.0 * (2 * n + 3)));
      t *= x / (2 * n + 3);
    }
    return;
  }
  const int N = nmax + 24 + (int)x;
  double ip1 = 0.0, in = 1e-250;
  const double xi = 1.0 / x;
  for (int n = N; n >= 1; n--) {
    const double im1 = (2 * n + 1) * xi * in + ip1;
    ip1 = in;
    in = im1;
    if (n - 1 <= nmax) v[(n - 1) * ST] = im1;
    if (fabs(in) > 1e250) {
      in *= 1e-250;
      ip1 *= 1e-250;
      for (int q = max(n - 1, 0); q <= nmax; q++) v[q * ST] *= 1e-250;
    }
  }
  const double sc = (sinh(x) / x) / v[0];
  for (int n = 0; n <= nmax; n++) v[n * ST] *= sc;
}

// k_n(x), n = 0..nmax, x > 0, normalised k_0 = (pi/2) e^{-x} / x (upward recurrence)
__device__ void sph_k(int nmax, double x, double* v) {
  const double e = 0.5 * M_PI * exp(-x);
  v[0] = e / x;
  if (nmax >= 1) v[1] = e * (1.0 / x + 1.0 / (x * x));
  for (int n = 1; n < nmax; n++) v[n + 1] = v[n - 1] + (2 * n + 1) / x * v[n];
}

// regular radial functions: j_n (Helmholtz) or i_n (Yukawa)
template <int ST>
__device__ __forceinline__ void radial_reg(int yuk, int nmax, double x, double* v) {
  if (yuk) sph_i<ST>(nmax, x, v);
  else sph_j<ST>(nmax, x, v);
}

// direction of v: cos(theta), and e^{i phi} (1 on the axis)
__device__ __forceinline__ void direction(double vx, double vy, double vz, double r, double& ct, double& st, double& cp,
                                          double& sp) {
  const double rxy = sqrt(vx * vx + vy * vy);
  if (r > 0) {
    ct = vz / r;
    st = rxy / r;
  } else {
    ct = 1.0;
    st = 0.0;
  }
  if (rxy > 0) {
    cp = vx / rxy;
    sp = vy / rxy;
  } else {
    cp = 1.0;
    sp = 0.0;
  }
}

// Ybar_m^m from Ybar_{m-1}^{m-1}
__device__ __forceinline__ double ybar_mm_next(int m, double st, double prev) {
  return sqrt((2.0 * m + 1.0) / (2.0 * m)) * st * prev;
}
// Ybar_n^m from Ybar_{n-1}^m, Ybar_{n-2}^m (n >= m+2)
__device__ __forceinline__ double ybar_next(int n, int m, double ct, double y1, double y2) {
  const double a = sqrt((4.0 * n * n - 1.0) / ((double)n * n - (double)m * m));
  const double b = sqrt((((double)n - 1) * (n - 1) - (double)m * m) / (4.0 * (n - 1) * (n - 1) - 1.0));
  return a * (ct * y1 - b * y2);
}

// Ybar_n^m(ct) for one (n, m), m >= 0
__device__ double ybar_one(int n, int m, double ct, double st) {
  double ymm = 0.28209479177387814;  // 1 / sqrt(4 pi)
  for (int k = 1; k <= m; k++) ymm = ybar_mm_next(k, st, ymm);
  if (n == m) return ymm;
  double y2 = ymm, y1 = sqrt(2.0 * m + 3.0) * ct * ymm;
  for (int l = m + 2; l <= n; l++) {
    const double y = ybar_next(l, m, ct, y1, y2);
    y2 = y1;
    y1 = y;
  }
  return y1;
}

struct Corner {  // root-cube corner (passed by value: the plan keeps it on the host)
  double x, y, z;
};

__device__ __forceinline__ void box_centre(int key, Corner bbox, double w, double& x, double& y, double& z) {
  int cx = 0, cy = 0, cz = 0;
  for (int i = 0; i < 10; i++) {
    cy |= ((key >> (3 * i)) & 1) << i;
    cx |= ((key >> (3 * i + 1)) & 1) << i;
    cz |= ((key >> (3 * i + 2)) & 1) << i;
  }
  x = bbox.x + (cx + 0.5) * w;
  y = bbox.y + (cy + 0.5) * w;
  z = bbox.z + (cz + 0.5) * w;
}

constexpr int kPts = 128;  // points per block of P2M and L2P

// What P2M and L2P need of a point relative to its box centre.
struct PointGeo {
  double ct, st, cp, sp;
};
// direction of v, and the radial functions of k|v| at jv[n kPts]
__device__ __forceinline__ PointGeo point_geo(int yuk, int p, double k, double vx, double vy, double vz, double* jv) {
  const double r = sqrt(vx * vx + vy * vy + vz * vz);
  PointGeo g;
  direction(vx, vy, vz, r, g.ct, g.st, g.cp, g.sp);
  radial_reg<kPts>(yuk, p, k * r, jv);
  return g;
}

__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// The recurrence coefficients of Ybar (ylm, [n (n+1) / 2 + m]): n = m: Ybar_m^m =
// x st Ybar_{m-1}^{m-1}; n = m + 1: x ct Ybar_m^m; above: x ct Ybar_{n-1}^m - y Ybar_{n-2}^m.

// ---------------------------------------------------------------- P2M
// One block (4 warps) per source leaf, 128 points at a time.
//   M_n^{+-m} = ik sum_j (j_n Ybar_n^m)(j) (q_j e^{-+i m phi_j})
// is for each order m a product of a (p + 1 - m) x points matrix and a points x
// 4 one (real and imaginary parts, both signs), done on the FP64 tensor
// instruction: the thread of a point leaves its radial functions in shared
// memory; then every warp takes orders of its own (dealt so that all have the
// same number of terms), evaluates the column of Ybar for 32 points at a time,
// one a lane, and multiplies.  (Before, a warp added each coefficient over its
// lanes with shuffles and computed a square root and a division for every
// term: 1,048,576 points at p = 16 took 2.3 ms; 0.74 now.)
constexpr int kMaxRow = kMaxP + 1;
constexpr int kPS = 36;  // row stride of a warp's staging: 32 points, conflict-free fragment reads

__global__ void __launch_bounds__(kPts) helm_p2m(int p, int K, double k, int yuk, const int* __restrict__ keys,
                                                 const int2* __restrict__ leaf, const float4* __restrict__ spos,
                                                 const float2* __restrict__ q, const double2* __restrict__ ylm,
                                                 Corner bbox, double w, double* __restrict__ M) {
  extern __shared__ double sm[];
  const int NT = (p + 1) * (p + 2) / 2;
  double* jv = sm;                            // [p + 1][kPts]
  double* geo = jv + (p + 1) * kPts;          // ct, st, cos phi, sin phi, Re q, Im q: [6][kPts]
  double* sum = geo + 6 * kPts;               // [terms, by order][4]
  double* mine = sum + 4 * NT + (threadIdx.x >> 5) * (kMaxRow + 3 + 4) * kPS;  // the warp's [24 rows][kPS], [4][kPS]
  double* wq = mine + (kMaxRow + 3) * kPS;
  const int b = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gq = lane >> 2, tq = lane & 3;
  for (int c = threadIdx.x; c < 4 * NT; c += kPts) sum[c] = 0.0;
  double xc, yc, zc;
  box_centre(keys[b], bbox, w, xc, yc, zc);
  const int2 lf = leaf[b];
  for (int base = 0; base < lf.y; base += kPts) {
    __syncthreads();  // the previous points are done with
    {
      const int i = base + threadIdx.x;
      double v[3] = {0.0, 0.0, 0.0};
      float2 qq = make_float2(0.f, 0.f);
      if (i < lf.y) {
        const float4 s = spos[lf.x + i];
        qq = q[lf.x + i];
        v[0] = (double)s.x - xc;
        v[1] = (double)s.y - yc;
        v[2] = (double)s.z - zc;
      }
      const PointGeo g = point_geo(yuk, p, k, v[0], v[1], v[2], jv + threadIdx.x);
      const double o[6] = {g.ct, g.st, g.cp, g.sp, qq.x, qq.y};
#pragma unroll
      for (int c = 0; c < 6; c++) geo[c * kPts + threadIdx.x] = o[c];
    }
    __syncthreads();
    const int nch = min(kPts, lf.y - base + 31) / 32;  // groups of 32 points
    double ymm[4], er[4], ei[4];                       // Ybar_m^m and e^{i m phi} of the lane's point of each group
#pragma unroll
    for (int ch = 0; ch < 4; ch++) {
      ymm[ch] = 0.28209479177387814;  // 1 / sqrt(4 pi)
      er[ch] = 1.0;
      ei[ch] = 0.0;
    }
    int row0 = 0;
    for (int m = 0; m <= p; row0 += p + 1 - m, m++) {
      if (m > 0) {
        const double xm = ylm[m * (m + 1) / 2 + m].x;
#pragma unroll
        for (int ch = 0; ch < 4; ch++) {
          if (ch >= nch) break;
          const int pt = 32 * ch + lane;
          const double cp = geo[2 * kPts + pt], sp = geo[3 * kPts + pt];
          ymm[ch] *= xm * geo[kPts + pt];
          const double t = er[ch] * cp - ei[ch] * sp;
          ei[ch] = er[ch] * sp + ei[ch] * cp;
          er[ch] = t;
        }
      }
      if (((m & 4) ? 3 - (m & 3) : (m & 3)) != warp) continue;  // another warp's order
      double acc[3][2] = {};
      const int nrow = p + 1 - m;
#pragma unroll
      for (int ch = 0; ch < 4; ch++) {
        if (ch >= nch) break;
        const int pt = 32 * ch + lane;
        const double ct = geo[pt], qr = geo[4 * kPts + pt], qi = geo[5 * kPts + pt];
        double y1 = ymm[ch], y2 = 0.0;
        __syncwarp();  // the previous group's reads are done
        mine[lane] = jv[m * kPts + pt] * y1;
        for (int n = m + 1; n <= p; n++) {
          const double2 c = ylm[n * (n + 1) / 2 + m];
          const double y = fma(c.x * ct, y1, -c.y * y2);
          y2 = y1;
          y1 = y;
          mine[(n - m) * kPS + lane] = jv[n * kPts + pt] * y;
        }
        wq[lane] = qr * er[ch] + qi * ei[ch];  // q e^{-i m phi}
        wq[kPS + lane] = qi * er[ch] - qr * ei[ch];
        wq[2 * kPS + lane] = qr * er[ch] - qi * ei[ch];  // q e^{+i m phi}
        wq[3 * kPS + lane] = qi * er[ch] + qr * ei[ch];
        __syncwarp();
#pragma unroll
        for (int k4 = 0; k4 < 32; k4 += 4) {
          const double bf = gq < 4 ? wq[gq * kPS + k4 + tq] : 0.0;
#pragma unroll
          for (int rt = 0; rt < 3; rt++)
            if (8 * rt < nrow) dmma884(acc[rt], mine[(8 * rt + gq) * kPS + k4 + tq], bf);
        }
      }
      if (tq < 2) {  // columns 2 tq, 2 tq + 1 of the four
#pragma unroll
        for (int rt = 0; rt < 3; rt++)
          if (8 * rt + gq < nrow) {
            sum[4 * (row0 + 8 * rt + gq) + 2 * tq] += acc[rt][0];
            sum[4 * (row0 + 8 * rt + gq) + 2 * tq + 1] += acc[rt][1];
          }
      }
    }
  }
  __syncthreads();
  double* out = M + (size_t)b * 2 * K;
  for (int c = threadIdx.x; c < K; c += kPts) {
    int n = 0;
    while ((n + 1) * (n + 1) <= c) n++;
    const int m = c - n * n - n, am = abs(m);
    const double* s = sum + 4 * (am * (p + 1) - am * (am - 1) / 2 + n - am) + (m < 0 ? 2 : 0);
    if (yuk) {  // (2 l / pi) (a + ib)
      out[c] = 2.0 * k / M_PI * s[0];
      out[K + c] = 2.0 * k / M_PI * s[1];
    } else {  // ik (a + ib) = -k b + i k a
      out[c] = -k * s[1];
      out[K + c] = k * s[0];
    }
  }
}

// ---------------------------------------------------------------- L2P
// One block per work item of up to 128 targets of a leaf, one thread per
// target: phi = sum L j_n(kr) Y_n^m, the recurrences' coefficients from the
// table (computed per term, a square root and a division each, the 1,048,576
// targets at p = 16 took 1.07 ms; 0.33 now).
__global__ void __launch_bounds__(kPts) helm_l2p(int p, int K, double k, int yuk, const int2* __restrict__ work,
                                                 const int* __restrict__ keys, const int2* __restrict__ leaf,
                                                 const float4* __restrict__ tpos, const double2* __restrict__ ylm,
                                                 Corner bbox, double w, const double* __restrict__ L,
                                                 double2* __restrict__ pot) {
  extern __shared__ double sm[];
  double* Ls = sm;               // [2K]
  double* jv = sm + 2 * K;       // [p + 1][kPts]
  const int2 wk = work[blockIdx.x];
  const int b = wk.x;
  for (int c = threadIdx.x; c < 2 * K; c += kPts) Ls[c] = L[(size_t)b * 2 * K + c];
  __syncthreads();
  double xc, yc, zc;
  box_centre(keys[b], bbox, w, xc, yc, zc);
  const int2 lf = leaf[b];
  const int i = wk.y + threadIdx.x;
  if (i >= lf.y) return;
  const float4 t = tpos[lf.x + i];
  jv += threadIdx.x;
  const PointGeo g = point_geo(yuk, p, k, (double)t.x - xc, (double)t.y - yc, (double)t.z - zc, jv);
  double pr = 0, pi = 0;
  double ymm = 0.28209479177387814, er = 1.0, ei = 0.0;
  for (int m = 0; m <= p; m++) {
    if (m > 0) {
      ymm *= ylm[m * (m + 1) / 2 + m].x * g.st;
      const double tt = er * g.cp - ei * g.sp;
      ei = er * g.sp + ei * g.cp;
      er = tt;
    }
    double y2 = 0.0, y1 = ymm;
    double ar = 0, ai = 0, br = 0, bi = 0;  // sums over n of L_n^m and L_n^-m
    for (int n = m; n <= p; n++) {
      if (n > m) {
        const double2 c = ylm[n * (n + 1) / 2 + m];
        const double y = fma(c.x * g.ct, y1, -c.y * y2);
        y2 = y1;
        y1 = y;
      }
      const double a = jv[n * kPts] * y1;
      const double* l = Ls + n * n + n;
      ar = fma(a, l[m], ar);
      ai = fma(a, l[K + m], ai);
      br = fma(a, l[-m], br);
      bi = fma(a, l[K - m], bi);
    }
    pr += ar * er - ai * ei;  // e^{i m phi}
    pi += ar * ei + ai * er;
    if (m > 0) {  // e^{-i m phi}
      pr += br * er + bi * ei;
      pi += bi * er - br * ei;
    }
  }
  pot[lf.x + i] = make_double2(pr, pi);
}

// ---------------------------------------------------------------- direct
__global__ void __launch_bounds__(128) helm_direct(int i0, int i1, const int* __restrict__ inv_i,
                                                   const float4* __restrict__ tpos, int nj,
                                                   const float4* __restrict__ spos, const float2* __restrict__ q,
                                                   double k, int yuk, double eps2, int excl,
                                                   double2* __restrict__ out) {
  __shared__ float4 sp[128];
  __shared__ float2 sq[128];
  const int i = i0 + blockIdx.x * blockDim.x + threadIdx.x;
  const bool act = i < i1;
  const float4 xi = tpos[act ? inv_i[i] : 0];
  double ar = 0, ai = 0;
  for (int j0 = 0; j0 < nj; j0 += 128) {
    __syncthreads();
    if (j0 + threadIdx.x < nj) {
      sp[threadIdx.x] = spos[j0 + threadIdx.x];
      sq[threadIdx.x] = q[j0 + threadIdx.x];
    }
    __syncthreads();
    const int nl = min(128, nj - j0);
    for (int jj = 0; jj < nl; jj++) {
      const double dx = (double)xi.x - sp[jj].x, dy = (double)xi.y - sp[jj].y, dz = (double)xi.z - sp[jj].z;
      const double d2 = dx * dx + dy * dy + dz * dz, r2 = d2 + eps2;
      if ((excl && d2 == 0.0) || r2 == 0.0) continue;
      const double r = sqrt(r2);
      double sn, cs;
      if (yuk) {
        sn = 0.0;
        cs = exp(-k * r);
      } else {
        sincos(k * r, &sn, &cs);
      }
      ar += (sq[jj].x * cs - sq[jj].y * sn) / r;
      ai += (sq[jj].x * sn + sq[jj].y * cs) / r;
    }
  }
  if (act) out[i - i0] = make_double2(0.25 / M_PI * ar, 0.25 / M_PI * ai);
}

// ---------------------------------------------------------------- operators
// (n, m) of row r of the parity images: (n, m > 0) by degree, O of them, then (n, 0)
__device__ __forceinline__ void row_order(int r, int O, int& n, int& m) {
  if (r >= O) {
    n = r - O;
    m = 0;
    return;
  }
  n = 1;
  while ((n + 1) * n / 2 <= r) n++;
  m = r - n * (n - 1) / 2 + 1;
}

// One block per (operator, source coefficient).  f = source basis function
// R_n(k|v|) Y_n^m(v^) at v = D + rad * s_q over the quadrature points s_q;
// g[i][m'] = sum_j f[i][j] e^{-i m' phi_j} 2 pi / NP;
// T[n'm'] = sum_i w_i g[i][m'] Ybar_n'^|m'|(x_i) / R'_n'(k rad).
// PAR: the M2L operators at azimuth 0 as the images of m2l_parity.cuh, T = A + iB
// combined over +-m' (rows) for columns (n, m >= 0): even block T_{m'm} +
// T_{-m'm}, odd block T_{m'm} - T_{-m'm}, halved for m' > 0 since the sum and
// difference of the two blocks' results give orders m' and -m'.
template <bool PAR>
__global__ void __launch_bounds__(256) helm_build_ops(int p, int K, double k, int yuk, const HelmOp* __restrict__ ops,
                                                      int NQ, int NP, const double* __restrict__ gl_x,
                                                      const double* __restrict__ gl_w,
                                                      const double* __restrict__ ybar_q,  // [NQ][P] Ybar at the nodes
                                                      double* __restrict__ opT, size_t ostride) {
  extern __shared__ double sm[];
  double2* f = (double2*)sm;                   // [NQ * NP]
  double2* g = f + (size_t)NQ * NP;            // [NQ][2p+1]
  double2* rt = g + (size_t)NQ * (2 * p + 1);  // [p+1] target radial values at rad
  const int o = blockIdx.y, c = blockIdx.x;
  const HelmOp op = ops[o];
  const int E = (p + 1) * (p + 2) / 2, O = p * (p + 1) / 2;
  int n = 0, m;
  if (PAR) {
    row_order(c, O, n, m);
  } else {
    while ((n + 1) * (n + 1) <= c) n++;
    m = c - n * n - n;
  }
  const int am = m < 0 ? -m : m;
  double rad[kMaxP + 1], rad2[kMaxP + 1];
  // 1. samples of the source basis function
  for (int t = threadIdx.x; t < NQ * NP; t += blockDim.x) {
    const int iq = t / NP, jq = t % NP;
    const double x = gl_x[iq], s = sqrt(fmax(0.0, 1.0 - x * x));
    double sphi, cphi;
    sincospi(2.0 * jq / NP, &sphi, &cphi);
    const double vx = op.dx + op.rad * s * cphi, vy = op.dy + op.rad * s * sphi, vz = op.dz + op.rad * x;
    const double r = sqrt(vx * vx + vy * vy + vz * vz);
    double ct, st, cp, sp;
    direction(vx, vy, vz, r, ct, st, cp, sp);
    const double yb = ybar_one(n, am, ct, st);
    // e^{i m phi}
    double er = 1.0, ei = 0.0;
    for (int l = 0; l < am; l++) {
      const double tt = er * cp - ei * sp;
      ei = er * sp + ei * cp;
      er = tt;
    }
    if (m < 0) ei = -ei;
    double rr, ri = 0.0;
    if (yuk) {  // k_n outgoing, i_n regular
      if (op.src_out) sph_k(n, k * r, rad);
      else sph_i(n, k * r, rad);
      rr = rad[n];
    } else {  // h_n = j_n + i y_n outgoing, j_n regular
      sph_j(n, k * r, rad);
      rr = rad[n];
      if (op.src_out) {
        sph_y(n, k * r, rad2);
        ri = rad2[n];
      }
    }
    // (rr + i ri) yb (er + i ei)
    f[t] = make_double2(yb * (rr * er - ri * ei), yb * (rr * ei + ri * er));
  }
  if (threadIdx.x == 0) {
    if (yuk) {
      if (op.tgt_out) sph_k(p, k * op.rad, rad);
      else sph_i(p, k * op.rad, rad);
      for (int l = 0; l <= p; l++) rt[l] = make_double2(rad[l], 0.0);
    } else {
      sph_j(p, k * op.rad, rad);
      if (op.tgt_out) sph_y(p, k * op.rad, rad2);
      for (int l = 0; l <= p; l++) rt[l] = make_double2(rad[l], op.tgt_out ? rad2[l] : 0.0);
    }
  }
  __syncthreads();
  // 2. azimuthal transform
  const int nm = 2 * p + 1;
  for (int t = threadIdx.x; t < NQ * nm; t += blockDim.x) {
    const int iq = t / nm, mp = t % nm - p;
    double sr = 0, si = 0;
    for (int jq = 0; jq < NP; jq++) {
      double sn, cs;
      sincospi(-2.0 * mp * jq / NP, &sn, &cs);
      const double2 v = f[iq * NP + jq];
      sr += v.x * cs - v.y * sn;
      si += v.x * sn + v.y * cs;
    }
    g[t] = make_double2(sr * (2.0 * M_PI / NP), si * (2.0 * M_PI / NP));
  }
  __syncthreads();
  // 3. polar transform, division by the target radial function, real form
  auto target = [&](int n2, int m2) -> double2 {
    const int am2 = m2 < 0 ? -m2 : m2;
    double sr = 0, si = 0;
    for (int iq = 0; iq < NQ; iq++) {
      const double wy = gl_w[iq] * ybar_q[(size_t)iq * ((p + 1) * (p + 2) / 2) + n2 * (n2 + 1) / 2 + am2];
      const double2 v = g[iq * nm + m2 + p];
      sr += wy * v.x;
      si += wy * v.y;
    }
    const double2 d = rt[n2];
    const double den = d.x * d.x + d.y * d.y;
    return make_double2((sr * d.x + si * d.y) / den, (si * d.x - sr * d.y) / den);
  };
  if (PAR) {
    const int te = parity_tiles(E), to = parity_tiles(O), nprod = yuk ? 1 : 3;
    const size_t se = parity_block(te), so = parity_block(to);
    double* img = opT + (size_t)o * ostride;
    for (int t = threadIdx.x; t < E; t += blockDim.x) {
      int n2, m2;
      row_order(t, O, n2, m2);
      double2 e = target(n2, m2), d = make_double2(0.0, 0.0);
      if (m2 > 0) {
        const double2 v = target(n2, -m2);
        d = make_double2(0.5 * (e.x - v.x), 0.5 * (e.y - v.y));
        e = make_double2(0.5 * (e.x + v.x), 0.5 * (e.y + v.y));
      }
      for (int pd = 0; pd < nprod; pd++) {  // A, -(A + B), B - A
        img[pd * se + parity_at(te, c, t)] = pd == 0 ? e.x : pd == 1 ? -(e.x + e.y) : e.y - e.x;
        if (t < O && c < O)
          img[nprod * se + pd * so + parity_at(to, c, t)] = pd == 0 ? d.x : pd == 1 ? -(d.x + d.y) : d.y - d.x;
      }
    }
    return;
  }
  double* col_re = opT + (size_t)o * ostride + (size_t)c * (2 * K);        // input re[c]
  double* col_im = opT + (size_t)o * ostride + (size_t)(K + c) * (2 * K);  // input im[c]
  for (int t = threadIdx.x; t < K; t += blockDim.x) {
    int n2 = 0;
    while ((n2 + 1) * (n2 + 1) <= t) n2++;
    const int m2 = t - n2 * n2 - n2;
    const double2 T = target(n2, m2);
    const double tr = T.x, ti = T.y;
    col_re[t] = tr;
    col_re[K + t] = ti;
    col_im[t] = -ti;
    col_im[K + t] = tr;
  }
}

// ---------------------------------------------------------------- glue
__global__ void helm_gather(int n, int nrhs, const int* __restrict__ perm, const float2* __restrict__ q,
                            float2* __restrict__ qs) {
  const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (t >= (size_t)n * nrhs) return;
  const int r = (int)(t / n), i = (int)(t % n);
  qs[t] = q[(size_t)r * n + perm[i]];
}

__global__ void helm_gather_real(int n, int nrhs, const int* __restrict__ perm, const float* __restrict__ q,
                                 float2* __restrict__ qs) {
  const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (t >= (size_t)n * nrhs) return;
  const int r = (int)(t / n), i = (int)(t % n);
  qs[t] = make_float2(q[(size_t)r * n + perm[i]], 0.f);
}

// real part of near + far, scaled, to caller order (Yukawa)
template <typename T>
__global__ void helm_finalize_real(int n, const int* __restrict__ perm, const double2* __restrict__ near,
                                   const double2* __restrict__ far, double scale, T* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[perm[i]] = (T)(scale * (near[i].x + (far ? far[i].x : 0.0)));
}

template <typename T>
__global__ void helm_finalize(int n, const int* __restrict__ perm, const double2* __restrict__ near,
                              const double2* __restrict__ far, T* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double2 a = near[i], b = far ? far[i] : make_double2(0.0, 0.0);
  const int o = perm[i];
  out[2 * (size_t)o] = (T)(a.x + b.x);
  out[2 * (size_t)o + 1] = (T)(a.y + b.y);
}

unsigned nb(size_t n, int t) { return (unsigned)((n + t - 1) / t); }

size_t helm_p2m_smem(int p) {
  return ((size_t)(p + 1 + 6) * kPts + 2 * (size_t)(p + 1) * (p + 2) + (kPts / 32) * (size_t)(kMaxRow + 3 + 4) * kPS) *
         sizeof(double);
}

}  // namespace

void launch_helm_gather(int n, int nrhs, const int* perm, const float* q, float* qs, cudaStream_t st) {
  if (n <= 0) return;
  helm_gather<<<nb((size_t)n * nrhs, 256), 256, 0, st>>>(n, nrhs, perm, (const float2*)q, (float2*)qs);
  FMMB_CHECK_LAUNCH();
}

void launch_helm_gather_real(int n, int nrhs, const int* perm, const float* q, float* qs, cudaStream_t st) {
  if (n <= 0) return;
  helm_gather_real<<<nb((size_t)n * nrhs, 256), 256, 0, st>>>(n, nrhs, perm, q, (float2*)qs);
  FMMB_CHECK_LAUNCH();
}

template <typename T>
void launch_helm_finalize_real(int n, const int* perm, const double* near, const double* far, double scale, T* out,
                               cudaStream_t st) {
  if (n <= 0) return;
  helm_finalize_real<T><<<nb(n, 256), 256, 0, st>>>(n, perm, (const double2*)near, (const double2*)far, scale, out);
  FMMB_CHECK_LAUNCH();
}
template void launch_helm_finalize_real<float>(int, const int*, const double*, const double*, double, float*,
                                               cudaStream_t);
template void launch_helm_finalize_real<double>(int, const int*, const double*, const double*, double, double*,
                                                cudaStream_t);

void launch_helm_p2m(int nleaf, int p, double k, bool yuk, const int* keys, const int2* leaf, const float4* spos,
                     const float* qs, const double* ylm, const float* bbox, double w, double* M, cudaStream_t st) {
  if (nleaf <= 0) return;
  const int K = (p + 1) * (p + 1);
  const Corner c{bbox[0], bbox[1], bbox[2]};  // host array
  helm_p2m<<<nleaf, kPts, helm_p2m_smem(p), st>>>(p, K, k, yuk ? 1 : 0, keys, leaf, spos, (const float2*)qs,
                                                  (const double2*)ylm, c, w, M);
  FMMB_CHECK_LAUNCH();
}

void launch_helm_l2p(int nwork, int p, double k, bool yuk, const int2* work, const int* keys, const int2* leaf,
                     const float4* tpos, const double* ylm, const float* bbox, double w, const double* L, double* pot,
                     cudaStream_t st) {
  if (nwork <= 0) return;
  const int K = (p + 1) * (p + 1);
  const Corner c{bbox[0], bbox[1], bbox[2]};  // host array
  helm_l2p<<<nwork, kPts, (2 * (size_t)K + (p + 1) * kPts) * sizeof(double), st>>>(
      p, K, k, yuk ? 1 : 0, work, keys, leaf, tpos, (const double2*)ylm, c, w, L, (double2*)pot);
  FMMB_CHECK_LAUNCH();
}

// The limit belongs to the function, not to a plan: one for every order, or a plan of
// a lower order would take it back under the others' launches.
void prepare_helm() {
  FMMB_CUDA(cudaFuncSetAttribute(helm_p2m, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)helm_p2m_smem(kMaxP)));
}

void launch_helm_direct(int i0, int i1, const int* inv_i, const float4* tpos, int nj, const float4* spos,
                        const float* qs, double k, bool yuk, double eps2, bool excl, double* out, cudaStream_t st) {
  if (i1 <= i0) return;
  helm_direct<<<nb(i1 - i0, 128), 128, 0, st>>>(i0, i1, inv_i, tpos, nj, spos, (const float2*)qs, k, yuk ? 1 : 0,
                                                eps2, excl ? 1 : 0, (double2*)out);
  FMMB_CHECK_LAUNCH();
}

template <typename T>
void launch_helm_finalize(int n, const int* perm, const double* near, const double* far, T* out, cudaStream_t st) {
  if (n <= 0) return;
  helm_finalize<T><<<nb(n, 256), 256, 0, st>>>(n, perm, (const double2*)near, (const double2*)far, out);
  FMMB_CHECK_LAUNCH();
}
template void launch_helm_finalize<float>(int, const int*, const double*, const double*, float*, cudaStream_t);
template void launch_helm_finalize<double>(int, const int*, const double*, const double*, double*, cudaStream_t);

size_t helm_build_smem(int p) {
  const int NQ = 2 * p + 8, NP = 2 * NQ;
  return ((size_t)NQ * NP + (size_t)NQ * (2 * p + 1) + (p + 1)) * sizeof(double2);
}

namespace {
template <bool PAR>
void build_ops(int p, double k, bool yuk, int nops, const HelmOp* ops, const double* gl_x, const double* gl_w,
               const double* ybar_q, double* opT, size_t ostride, cudaStream_t st) {
  if (nops <= 0) return;
  const int K = (p + 1) * (p + 1), NQ = 2 * p + 8, NP = 2 * NQ;
  const size_t smem = helm_build_smem(p);
  FMMB_CUDA(cudaFuncSetAttribute(helm_build_ops<PAR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)helm_build_smem(kMaxP)));
  for (int o0 = 0; o0 < nops; o0 += 65535) {
    dim3 grid(PAR ? (p + 1) * (p + 2) / 2 : K, std::min(65535, nops - o0));
    helm_build_ops<PAR><<<grid, 256, smem, st>>>(p, K, k, yuk ? 1 : 0, ops + o0, NQ, NP, gl_x, gl_w, ybar_q,
                                                 opT + (size_t)o0 * ostride, ostride);
    FMMB_CHECK_LAUNCH();
  }
}
}  // namespace

void launch_helm_build_ops(int p, double k, bool yuk, int nops, const HelmOp* ops, const double* gl_x,
                           const double* gl_w, const double* ybar_q, double* opT, cudaStream_t st) {
  const size_t K = (size_t)(p + 1) * (p + 1);
  build_ops<false>(p, k, yuk, nops, ops, gl_x, gl_w, ybar_q, opT, 4 * K * K, st);
}

void launch_helm_build_parity(int p, double k, bool yuk, int nops, const HelmOp* ops, const double* gl_x,
                              const double* gl_w, const double* ybar_q, double* img, size_t stride, cudaStream_t st) {
  build_ops<true>(p, k, yuk, nops, ops, gl_x, gl_w, ybar_q, img, stride, st);
}

}  // namespace fmmb
