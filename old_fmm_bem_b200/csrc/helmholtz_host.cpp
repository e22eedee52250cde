// Host side of the complex Helmholtz kernel (FMMB_HELMHOLTZ_G): the per-level
// translation operators (built on the GPU by helmholtz.cu) and the pair jobs
// that apply them with the FP64 pair kernel.  Called by fmmb_set_geometry
// after the octree is built; the evaluation itself is in api.cpp.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <vector>

#include "internal.h"
#include "kernels.h"

namespace fmmb {
namespace {

// Gauss-Legendre nodes and weights on [-1, 1] (Newton on P_n from the
// Chebyshev guesses)
void gauss_legendre(int n, std::vector<double>& x, std::vector<double>& w) {
  x.assign(n, 0.0);
  w.assign(n, 0.0);
  for (int i = 0; i < n; i++) {
    double z = std::cos(M_PI * (i + 0.75) / (n + 0.5)), dp = 1.0;
    for (int it = 0; it < 100; it++) {
      double p0 = 1.0, p1 = z;
      for (int k = 2; k <= n; k++) {
        const double p2 = ((2.0 * k - 1.0) * z * p1 - (k - 1.0) * p0) / k;
        p0 = p1;
        p1 = p2;
      }
      dp = n * (z * p1 - p0) / (z * z - 1.0);
      const double dz = p1 / dp;
      z -= dz;
      if (std::fabs(dz) < 1e-16) break;
    }
    {
      double p0 = 1.0, p1 = z;
      for (int k = 2; k <= n; k++) {
        const double p2 = ((2.0 * k - 1.0) * z * p1 - (k - 1.0) * p0) / k;
        p0 = p1;
        p1 = p2;
      }
      dp = n * (z * p1 - p0) / (z * z - 1.0);
    }
    x[i] = z;
    w[i] = 2.0 / ((1.0 - z * z) * dp * dp);
  }
}

// Ybar_n^m(x), m >= 0, the fully normalised recurrence of helmholtz.cu,
// [n (n+1) / 2 + m]
void ybar_table(int p, double x, double* out) {
  const double s = std::sqrt(std::max(0.0, 1.0 - x * x));
  double ymm = 0.28209479177387814;
  for (int m = 0; m <= p; m++) {
    if (m > 0) ymm = std::sqrt((2.0 * m + 1.0) / (2.0 * m)) * s * ymm;
    double y2 = 0.0, y1 = ymm;
    for (int n = m; n <= p; n++) {
      double y;
      if (n == m) {
        y = ymm;
      } else if (n == m + 1) {
        y = std::sqrt(2.0 * m + 3.0) * x * ymm;
      } else {
        const double a = std::sqrt((4.0 * n * n - 1.0) / ((double)n * n - (double)m * m));
        const double b = std::sqrt((((double)n - 1) * (n - 1) - (double)m * m) / (4.0 * (n - 1) * (n - 1) - 1.0));
        y = a * (x * y1 - b * y2);
      }
      if (n > m) {
        y2 = y1;
        y1 = y;
      }
      out[n * (n + 1) / 2 + m] = y;
    }
  }
}

template <typename T>
void upload_vec(DevBuf<T>& d, const std::vector<T>& h) {
  d.alloc(h.size());
  if (!h.empty()) FMMB_CUDA(cudaMemcpy(d.get(), h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
}

}  // namespace

void helm_setup(fmmb_plan* pl) {
  const int p = pl->p, K = pl->K, lmax = pl->lmax;
  const double k = pl->cfg.wavenumber, rd = pl->bbox[3];
  cudaStream_t s = pl->st.main;
  auto width = [&](int l) { return rd / (double)(1 << l); };
  // operators: M2M for child levels 3..lmax (8 octants each), L2L likewise
  std::vector<HelmOp> ops;
  auto octant_offset = [&](int oct, double wc, double* o) {  // child centre - parent centre
    o[0] = (((oct >> 1) & 1) - 0.5) * wc;  // key bit 1: x
    o[1] = ((oct & 1) - 0.5) * wc;         // key bit 0: y
    o[2] = (((oct >> 2) & 1) - 0.5) * wc;  // key bit 2: z
  };
  const bool yuk = pl->cfg.kernel == FMMB_YUKAWA;
  // Helmholtz: keeps k * rad below the first zero of j_0 (i_n of Yukawa has no zeros)
  const double rad_cap = yuk ? 1e300 : 2.5 / k;
  pl->hop_m2m0 = 0;
  for (int lc = 3; lc <= lmax; lc++)
    for (int oct = 0; oct < 8; oct++) {
      double o[3];
      octant_offset(oct, width(lc), o);
      ops.push_back({-o[0], -o[1], -o[2], 2.0 * width(lc - 1), 1, 1});
    }
  pl->hop_l2l0 = (int)ops.size();
  for (int lc = 3; lc <= lmax; lc++)
    for (int oct = 0; oct < 8; oct++) {
      double o[3];
      octant_offset(oct, width(lc), o);
      ops.push_back({o[0], o[1], o[2], std::min(0.8660254037844386 * width(lc), rad_cap), 0, 0});
    }
  // M2L: levels 2..lmax x the 61 classes, at azimuth 0
  std::vector<HelmOp> mops;
  for (int l = 2; l <= lmax; l++)
    for (const auto& g : pl->ops.cls_geom) {
      const double w = width(l);
      mops.push_back({std::sqrt((double)g[0]) * w, 0.0, g[1] * w, std::min(0.8660254037844386 * w, rad_cap), 1, 0});
    }
  const int nops = (int)ops.size();
  const size_t ostride = (size_t)4 * K * K;
  pl->d_hops.alloc((size_t)nops * ostride);
  {
    const int NQ = 2 * p + 8, P = (p + 1) * (p + 2) / 2;
    std::vector<double> gx, gw;
    gauss_legendre(NQ, gx, gw);
    std::vector<double> yb((size_t)NQ * P);
    for (int i = 0; i < NQ; i++) ybar_table(p, gx[i], yb.data() + (size_t)i * P);
    DevBuf<double> d_gx, d_gw, d_yb;
    DevBuf<HelmOp> d_ops, d_mops;
    upload_vec(d_gx, gx);
    upload_vec(d_gw, gw);
    upload_vec(d_yb, yb);
    upload_vec(d_ops, ops);
    launch_helm_build_ops(p, k, yuk, nops, d_ops.get(), d_gx.get(), d_gw.get(), d_yb.get(), pl->d_hops.get(), s);
    const size_t pstride = parity_img_stride(yuk ? 2 : 1, p);
    pl->d_par.alloc(mops.size() * pstride);
    FMMB_CUDA(cudaMemsetAsync(pl->d_par.get(), 0, mops.size() * pstride * sizeof(double), s));  // the padding stays zero
    upload_vec(d_mops, mops);
    launch_helm_build_parity(p, k, yuk, (int)mops.size(), d_mops.get(), d_gx.get(), d_gw.get(), d_yb.get(),
                             pl->d_par.get(), pstride, s);
    FMMB_CUDA(cudaStreamSynchronize(s));
  }
  int nsm = 148;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, pl->device);
  pl->nsm = nsm;
  prepare_translate_pairs_f64();
  build_pair_jobs(pl, pl->hop_m2m0, pl->hop_l2l0, 8, s);
  prepare_m2l_parity(yuk ? 2 : 1, p);
  build_parity_job(pl, s);
  // near-field work items and the inverse target permutation of the direct sum
  build_work_dev(pl, false, s);
  build_inverse_perm_dev(pl, s);
  // recurrence coefficients of Ybar
  std::vector<double> ylm((size_t)(p + 1) * (p + 2), 0.0);
  for (int n = 0; n <= p; n++)
    for (int m = 0; m <= n; m++) {
      double* c = &ylm[(size_t)(n * (n + 1) / 2 + m) * 2];
      if (n == m) {
        c[0] = m ? std::sqrt((2.0 * m + 1.0) / (2.0 * m)) : 1.0;
      } else if (n == m + 1) {
        c[0] = std::sqrt(2.0 * m + 3.0);
      } else {
        const double a = std::sqrt((4.0 * n * n - 1.0) / ((double)n * n - (double)m * m));
        c[0] = a;
        c[1] = a * std::sqrt((((double)n - 1) * (n - 1) - (double)m * m) / (4.0 * (n - 1) * (n - 1) - 1.0));
      }
    }
  upload_vec(pl->d_ylm, ylm);
  prepare_helm();
  const int nr = pl->cfg.nrhs;
  pl->qs.alloc((size_t)2 * pl->nj * nr);
  pl->M.alloc((size_t)pl->tot_j * 2 * K);
  pl->L.alloc((size_t)pl->tot_i * 2 * K);
  pl->pot_s.alloc((size_t)4 * pl->ni);  // near, far (complex)
  pl->use_tc = false;
  pl->use_h16 = false;
  FMMB_CUDA(cudaStreamSynchronize(s));
}

}  // namespace fmmb
