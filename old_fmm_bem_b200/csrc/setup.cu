// Device-side construction of the evaluation work lists of a geometry
// (fmmb_set_geometry): the tensor-core M2L's pair tiles and the CSR of its
// per-box reduction, the near-field work items, the inverse target
// permutation.  Scans and stable radix sorts (tree.cu) over the device lists
// the tree build produced, so that none of it is copied to the host; the
// results are the ones the former host loops gave (same orders, ties kept in
// input order).
//
// The lists restate the work of the reference's fmm() driver
// (fmm/fmm.cxx:29-152: ijbox's lists per level, kernel/m2l.cxx:13-93 over
// them) in the order the kernels want it.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <vector>

#include "internal.h"
#include "kernels.h"

namespace fmmb {
namespace {

constexpr int kT = 256;
constexpr int kMaxLev = 12;

inline unsigned nblk(long long n, int t) { return (unsigned)((n + t - 1) / t); }
inline int bits_for(long long n) {  // bits to hold values in [0, n)
  int b = 1;
  while ((1LL << b) < n) b++;
  return b;
}

// The (level, box, slot) enumeration of the M2L pairs: levels 2..lmax
// ascending, boxes of a level in order, the 189 slots of a box in order.
struct LevTab {
  int nlev;                // levels 2..lmax
  int vstart[kMaxLev + 1]; // first virtual index of level lev - 2 (vstart[nlev] = total)
  int boxoff[kMaxLev];     // first box of the level in the all-level target arrays
  int srcoff[kMaxLev];     // first box of the level in the all-level source arrays
  int set[kMaxLev];        // operator set of the level
};

__device__ __forceinline__ void lev_of(const LevTab& T, int v, int& l, int& b, int& sl) {
  l = 0;
  while (l + 1 < T.nlev && T.vstart[l + 1] <= v) l++;
  const int r = v - T.vstart[l];
  b = r / kM2LSlots;
  sl = r - b * kM2LSlots;
}

__global__ void m2l_pair_flags(int V, LevTab T, const int* __restrict__ lst, int* __restrict__ flag) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= V) return;
  int l, b, sl;
  lev_of(T, v, l, b, sl);
  flag[v] = lst[(size_t)(T.boxoff[l] + b) * kM2LSlots + sl] >= 0 ? 1 : 0;
}

// pair k (in enumeration order) -> operator key, source row, target row and,
// when wanted, azimuth index of the relative position; `per` operators a set
__global__ void m2l_pair_emit(int V, LevTab T, const int* __restrict__ lst, const int* __restrict__ key_i,
                              const int* __restrict__ slot_rel, const int* __restrict__ rel_to_op, int per,
                              const int* __restrict__ pos, int* __restrict__ opk, int* __restrict__ ord,
                              int* __restrict__ src, int* __restrict__ dst, int* __restrict__ phi) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= V) return;
  int l, b, sl;
  lev_of(T, v, l, b, sl);
  const int box = T.boxoff[l] + b;
  const int s = lst[(size_t)box * kM2LSlots + sl];
  if (s < 0) return;
  const int k = pos[v];
  const int rel = slot_rel[(key_i[box] & 7) * kM2LSlots + sl];
  opk[k] = T.set[l] * per + rel_to_op[rel];
  if (phi) phi[k] = rel / 7;
  ord[k] = k;
  src[k] = T.srcoff[l] + s;
  dst[k] = box;
}

__global__ void count_keys(int n, const int* __restrict__ key, int* __restrict__ cnt) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n) atomicAdd(&cnt[key[j]], 1);
}

__global__ void tiles_per_key(int nk, int tt, const int* __restrict__ cnt, int* __restrict__ tiles) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o < nk) tiles[o] = (cnt[o] + tt - 1) / tt;
}

// sorted pair j -> tile tile_base[op] + r / tt, column r % tt (r = its rank
// among the pairs of its operator)
__global__ void fill_tiles(int n, int tt, const int* __restrict__ opk, const int* __restrict__ ord,
                           const int* __restrict__ src, const int* __restrict__ dst, const int* __restrict__ phi,
                           const int* __restrict__ op_start, const int* __restrict__ tile_base,
                           int* __restrict__ tile_op, int* __restrict__ tile_src, int* __restrict__ tdst,
                           int* __restrict__ tile_phi) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int op = opk[j], r = j - op_start[op];
  const int t = tile_base[op] + r / tt, c = r % tt;
  tile_src[(size_t)t * tt + c] = src[ord[j]];
  tdst[(size_t)t * tt + c] = dst[ord[j]];
  if (phi) tile_phi[(size_t)t * tt + c] = phi[ord[j]];
  if (c == 0) tile_op[t] = op;
}

__global__ void fill_tile_y(int ntile, int* __restrict__ ty) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntile) return;
  ty[2 * t] = t * 128;
  ty[2 * t + 1] = 0;
}

__global__ void nonneg_flags(int n, const int* __restrict__ a, int* __restrict__ flag) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) flag[k] = a[k] >= 0 ? 1 : 0;
}

// column k of the tiles with a target -> (target row, k), in k order
__global__ void compact_cols(int n, const int* __restrict__ tdst, const int* __restrict__ pos,
                             int* __restrict__ rowk, int* __restrict__ colk) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n || tdst[k] < 0) return;
  rowk[pos[k]] = tdst[k];
  colk[pos[k]] = k;
}

__global__ void run_starts(int n, const int* __restrict__ key, int* __restrict__ flag) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m < n) flag[m] = (m == 0 || key[m] != key[m - 1]) ? 1 : 0;
}

__global__ void emit_runs(int n, const int* __restrict__ key, const int* __restrict__ pos, int* __restrict__ rows,
                          int* __restrict__ ptr) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= n) return;
  const bool st = m == 0 || key[m] != key[m - 1];  // pos[m]: the runs started before m
  if (st) {
    rows[pos[m]] = key[m];
    ptr[pos[m]] = m;
  }
  if (m == n - 1) ptr[pos[m] + (st ? 1 : 0)] = n;
}

// ---- near-field work items ----
__global__ void leaf_item_counts(int nleaf, const int2* __restrict__ leaf_i, const int2* __restrict__ leaf_j,
                                 const int* __restrict__ list, int* __restrict__ cnt, long long* __restrict__ nsrc) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nleaf) return;
  long long s = 0;
  for (int sl = 0; sl < kP2PSlots; sl++) {
    const int jl = list[(size_t)b * kP2PSlots + sl];
    if (jl >= 0) s += leaf_j[jl].y;
  }
  nsrc[b] = s > 0 ? s : 1;
  cnt[b] = (leaf_i[b].y + 127) / 128;
}

// items of leaf b in leaf order; the sort key puts the heaviest first
__global__ void leaf_items(int nleaf, const int2* __restrict__ leaf_i, const long long* __restrict__ nsrc,
                           const int* __restrict__ base, int2* __restrict__ work, int* __restrict__ skey,
                           int* __restrict__ sval) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nleaf) return;
  const int n = leaf_i[b].y;
  for (int t = 0, k = base[b]; t < n; t += 128, k++) {
    const long long cost = (long long)min(128, n - t) * nsrc[b];
    const long long cap = (1LL << 30) - 1;
    work[k] = make_int2(b, t);
    skey[k] = (int)(cap - (cost < cap ? cost : cap));
    sval[k] = k;
  }
}

// ---- P2M work items: pieces of up to `per` sources of a source leaf ----
__global__ void src_item_counts(int nleaf, int per, const int2* __restrict__ leaf_j, int* __restrict__ cnt) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < nleaf) cnt[b] = (leaf_j[b].y + per - 1) / per;
}

__global__ void src_items(int nleaf, int per, const int2* __restrict__ leaf_j, const int* __restrict__ base,
                          int2* __restrict__ work) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nleaf) return;
  const int n = leaf_j[b].y;
  for (int t = 0, k = base[b]; t < n; t += per, k++) work[k] = make_int2(b, t);
}

// sorted item j -> launch (j & 1), position j >> 1 within it
__global__ void deal_items(int n, int n0, const int* __restrict__ sorted, const int2* __restrict__ work,
                           int2* __restrict__ out) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  out[(j & 1) ? n0 + (j >> 1) : (j >> 1)] = work[sorted[j]];
}

__global__ void invert_perm(int n, const int* __restrict__ perm, int* __restrict__ inv) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) inv[perm[i]] = i;
}

int d2h_int(const int* p, cudaStream_t s) {
  int h = 0;
  FMMB_CUDA(cudaMemcpyAsync(&h, p, sizeof(int), cudaMemcpyDeviceToHost, s));
  FMMB_CUDA(cudaStreamSynchronize(s));
  return h;
}

}  // namespace

namespace {

// The M2L pairs of levels 2..lmax sorted by operator, in tiles of tt pairs:
// the operator of pair (level, relative position r) is set(level) * per +
// rel_to_op[r].  phi (may be null): the azimuth index of each pair.  False when
// the enumeration does not fit an int.
struct M2LTiles {
  int npair = 0, ntile = 0;
};
bool build_m2l_tiles(fmmb_plan* pl, bool sets, int per, const int* rel_to_op, int tt, DevBuf<int>& tile_op,
                     DevBuf<int>& tile_src, DevBuf<int>* tile_phi, M2LTiles& out, TmpBuf<int>& tdst, cudaStream_t s) {
  const int lmax = pl->lmax;
  if (lmax - 1 > kMaxLev) return false;
  LevTab T{};
  long long V = 0;
  T.nlev = 0;
  for (int lev = 2; lev <= lmax; lev++) {
    const int l = T.nlev++;
    T.vstart[l] = (int)V;
    T.boxoff[l] = pl->off_i[lev];
    T.srcoff[l] = pl->off_j[lev];
    T.set[l] = sets ? lev - 2 : 0;
    V += (long long)pl->nbox_i[lev] * kM2LSlots;
    if (V >= (1LL << 31) - 1) return false;  // the host loops take such sizes
  }
  T.vstart[T.nlev] = (int)V;
  const int nv = (int)V;
  const int nops = (sets ? lmax - 1 : 1) * per;
  TmpBuf<int> pos(s);
  pos.alloc((size_t)nv + 1);
  m2l_pair_flags<<<nblk(nv, kT), kT, 0, s>>>(nv, T, pl->m2l_list.get(), pos.get());
  FMMB_CHECK_LAUNCH();
  FMMB_CUDA(cudaMemsetAsync(pos.get() + nv, 0, sizeof(int), s));
  exclusive_scan(pos.get(), nv + 1, s);
  const int npair = d2h_int(pos.get() + nv, s);
  TmpBuf<int> opk(s), ord(s), src(s), dst(s), phi(s);
  opk.alloc(npair);
  ord.alloc(npair);
  src.alloc(npair);
  dst.alloc(npair);
  if (tile_phi) phi.alloc(npair);
  m2l_pair_emit<<<nblk(nv, kT), kT, 0, s>>>(nv, T, pl->m2l_list.get(), pl->key_i.get(), pl->d_slot_rel.get(),
                                           rel_to_op, per, pos.get(), opk.get(), ord.get(), src.get(), dst.get(),
                                           tile_phi ? phi.get() : nullptr);
  FMMB_CHECK_LAUNCH();
  radix_sort(opk.get(), ord.get(), npair, bits_for(nops), s);  // stable: enumeration order within an operator
  // tiles of tt pairs per operator
  TmpBuf<int> cnt(s), op_start(s), tile_base(s);
  cnt.alloc(nops + 1);
  op_start.alloc(nops + 1);
  tile_base.alloc(nops + 1);
  FMMB_CUDA(cudaMemsetAsync(cnt.get(), 0, (nops + 1) * sizeof(int), s));
  if (npair > 0) {
    count_keys<<<nblk(npair, kT), kT, 0, s>>>(npair, opk.get(), cnt.get());
    FMMB_CHECK_LAUNCH();
  }
  FMMB_CUDA(cudaMemcpyAsync(op_start.get(), cnt.get(), (nops + 1) * sizeof(int), cudaMemcpyDeviceToDevice, s));
  tiles_per_key<<<nblk(nops + 1, kT), kT, 0, s>>>(nops + 1, tt, cnt.get(), tile_base.get());
  FMMB_CHECK_LAUNCH();
  exclusive_scan(op_start.get(), nops + 1, s);
  exclusive_scan(tile_base.get(), nops + 1, s);
  const int ntile = d2h_int(tile_base.get() + nops, s);
  const size_t ncol = (size_t)std::max(ntile, 1) * tt;
  tile_op.alloc(std::max(ntile, 1));
  tile_src.alloc(ncol);
  tdst.alloc(ncol);
  FMMB_CUDA(cudaMemsetAsync(tile_src.get(), 0xff, ncol * sizeof(int), s));
  FMMB_CUDA(cudaMemsetAsync(tdst.get(), 0xff, ncol * sizeof(int), s));
  if (tile_phi) {
    tile_phi->alloc(ncol);
    FMMB_CUDA(cudaMemsetAsync(tile_phi->get(), 0, ncol * sizeof(int), s));
  }
  if (npair > 0) {
    fill_tiles<<<nblk(npair, kT), kT, 0, s>>>(npair, tt, opk.get(), ord.get(), src.get(), dst.get(),
                                             tile_phi ? phi.get() : nullptr, op_start.get(), tile_base.get(),
                                             tile_op.get(), tile_src.get(), tdst.get(),
                                             tile_phi ? tile_phi->get() : nullptr);
    FMMB_CHECK_LAUNCH();
  }
  out.npair = npair;
  out.ntile = ntile;
  return true;
}

}  // namespace

void build_parity_job(fmmb_plan* pl, cudaStream_t s) {
  const int ncls = (int)pl->ops.cls_geom.size();
  const bool helm = helm_family(pl->cfg.kernel), sets = helm || pl->ref;
  fmmb_plan::PairJob& job = pl->par_m2l;
  M2LTiles t;
  TmpBuf<int> tdst(s);
  if (build_m2l_tiles(pl, sets, ncls, pl->d_rel_to_cls.get(), 32, job.tile_op, job.tile_src, &job.tile_phi, t, tdst, s)) {
    job.tile_dst.alloc((size_t)std::max(t.ntile, 1) * 32);
    FMMB_CUDA(cudaMemcpyAsync(job.tile_dst.get(), tdst.get(), (size_t)t.ntile * 32 * sizeof(int), cudaMemcpyDeviceToDevice, s));
    FMMB_CUDA(cudaStreamSynchronize(s));
    job.ntile = t.ntile;
    job.tp = 32;
    return;
  }
  // more box slots than an int enumerates: the same lists on the host
  std::vector<int> key(pl->tot_i), lst((size_t)pl->tot_i * kM2LSlots);
  FMMB_CUDA(cudaMemcpy(key.data(), pl->key_i.get(), key.size() * sizeof(int), cudaMemcpyDeviceToHost));
  FMMB_CUDA(cudaMemcpy(lst.data(), pl->m2l_list.get(), lst.size() * sizeof(int), cudaMemcpyDeviceToHost));
  std::vector<std::vector<std::array<int, 3>>> by((size_t)(sets ? pl->lmax - 1 : 1) * ncls);
  for (int lev = 2; lev <= pl->lmax; lev++)
    for (int b = 0; b < pl->nbox_i[lev]; b++) {
      const int box = pl->off_i[lev] + b;
      for (int sl = 0; sl < kM2LSlots; sl++) {
        const int src = lst[(size_t)box * kM2LSlots + sl];
        if (src < 0) continue;
        const int rel = pl->ops.slot_rel[(key[box] & 7) * kM2LSlots + sl];
        by[(size_t)(sets ? lev - 2 : 0) * ncls + pl->ops.rel_to_cls[rel]].push_back({pl->off_j[lev] + src, box, rel / 7});
      }
    }
  std::vector<int> top, col[3];
  for (size_t o = 0; o < by.size(); o++)
    for (size_t k = 0; k < by[o].size(); k += 32) {
      top.push_back((int)o);
      for (size_t c = k; c < k + 32; c++)
        for (int w = 0; w < 3; w++) col[w].push_back(c < by[o].size() ? by[o][c][w] : (w == 2 ? 0 : -1));
    }
  auto up = [](DevBuf<int>& d, const std::vector<int>& h) {
    d.alloc(h.size());
    if (!h.empty()) FMMB_CUDA(cudaMemcpy(d.get(), h.data(), h.size() * sizeof(int), cudaMemcpyHostToDevice));
  };
  up(job.tile_op, top);
  up(job.tile_src, col[0]);
  up(job.tile_dst, col[1]);
  up(job.tile_phi, col[2]);
  job.ntile = (int)top.size();
  job.tp = 32;
}

bool build_m2l_job_dev(fmmb_plan* pl, fmmb_plan::TcJob& job, int ys, cudaStream_t s) {
  M2LTiles t;
  TmpBuf<int> tdst(s);
  if (!build_m2l_tiles(pl, pl->ops.m2l_sets > 1, 316, pl->d_rel_to_op.get(), 128, job.tile_op, job.tile_src, nullptr, t,
                       tdst, s))
    return false;
  const int npair = t.npair, ntile = t.ntile;
  job.ntile = ntile;
  job.tile_y.alloc((size_t)std::max(ntile, 1) * 2);
  if (ntile > 0) {
    fill_tile_y<<<nblk(ntile, kT), kT, 0, s>>>(ntile, job.tile_y.get());
    FMMB_CHECK_LAUNCH();
  }
  // per output box, its pair rows (tile * 128 + column) in increasing order
  const int ncol = ntile * 128;
  TmpBuf<int> cpos(s);
  cpos.alloc((size_t)ncol + 1);
  if (ncol > 0) {
    nonneg_flags<<<nblk(ncol, kT), kT, 0, s>>>(ncol, tdst.get(), cpos.get());
    FMMB_CHECK_LAUNCH();
  }
  FMMB_CUDA(cudaMemsetAsync(cpos.get() + ncol, 0, sizeof(int), s));
  exclusive_scan(cpos.get(), ncol + 1, s);
  TmpBuf<int> rowk(s), colk(s);
  rowk.alloc(std::max(npair, 1));
  colk.alloc(std::max(npair, 1));
  if (ncol > 0) {
    compact_cols<<<nblk(ncol, kT), kT, 0, s>>>(ncol, tdst.get(), cpos.get(), rowk.get(), colk.get());
    FMMB_CHECK_LAUNCH();
  }
  radix_sort(rowk.get(), colk.get(), npair, bits_for(pl->tot_i), s);
  TmpBuf<int> rpos(s);
  rpos.alloc((size_t)npair + 1);
  if (npair > 0) {
    run_starts<<<nblk(npair, kT), kT, 0, s>>>(npair, rowk.get(), rpos.get());
    FMMB_CHECK_LAUNCH();
  }
  FMMB_CUDA(cudaMemsetAsync(rpos.get() + npair, 0, sizeof(int), s));
  exclusive_scan(rpos.get(), npair + 1, s);
  const int nred = d2h_int(rpos.get() + npair, s);
  job.nred = nred;
  job.red_rows.alloc(std::max(nred, 1));
  job.red_ptr.alloc((size_t)nred + 1);
  if (npair > 0) {
    emit_runs<<<nblk(npair, kT), kT, 0, s>>>(npair, rowk.get(), rpos.get(), job.red_rows.get(), job.red_ptr.get());
    FMMB_CHECK_LAUNCH();
  } else {
    FMMB_CUDA(cudaMemsetAsync(job.red_ptr.get(), 0, sizeof(int), s));
  }
  job.red_idx.alloc(std::max(npair, 1));
  if (npair > 0)
    FMMB_CUDA(cudaMemcpyAsync(job.red_idx.get(), colk.get(), (size_t)npair * sizeof(int), cudaMemcpyDeviceToDevice, s));
  job.ys = ys;
  pl->tc_y.alloc((size_t)std::max(ntile, 1) * 128 * ys);
  FMMB_CUDA(cudaStreamSynchronize(s));
  return true;
}

void build_p2p_work_dev(fmmb_plan* pl, cudaStream_t s) {
  const int nleaf = pl->nbox_i[pl->lmax];
  TmpBuf<int> cnt(s);
  TmpBuf<long long> nsrc(s);
  cnt.alloc((size_t)nleaf + 1);
  nsrc.alloc(std::max(nleaf, 1));
  FMMB_CUDA(cudaMemsetAsync(cnt.get() + nleaf, 0, sizeof(int), s));
  if (nleaf > 0) {
    leaf_item_counts<<<nblk(nleaf, kT), kT, 0, s>>>(nleaf, pl->leaf_i.get(), pl->leaf_j.get(), pl->p2p_list.get(),
                                                   cnt.get(), nsrc.get());
    FMMB_CHECK_LAUNCH();
  }
  exclusive_scan(cnt.get(), nleaf + 1, s);
  const int n = d2h_int(cnt.get() + nleaf, s);
  pl->m_p2p_work.alloc(std::max(n, 1));
  pl->m_p2p_nwork = n;
  TmpBuf<int> skey(s), sval(s);
  skey.alloc(std::max(n, 1));
  sval.alloc(std::max(n, 1));
  if (nleaf > 0) {
    leaf_items<<<nblk(nleaf, kT), kT, 0, s>>>(nleaf, pl->leaf_i.get(), nsrc.get(), cnt.get(), pl->m_p2p_work.get(),
                                             skey.get(), sval.get());
    FMMB_CHECK_LAUNCH();
  }
  radix_sort(skey.get(), sval.get(), n, 30, s);  // stable: leaf order among equal costs
  const int n0 = (n + 1) / 2;
  pl->p2p_work.alloc(std::max(n, 1));
  if (n > 0) {
    deal_items<<<nblk(n, kT), kT, 0, s>>>(n, n0, sval.get(), pl->m_p2p_work.get(), pl->p2p_work.get());
    FMMB_CHECK_LAUNCH();
  }
  pl->p2p_nwork = n;
  pl->p2p_nwork0 = n0;
  FMMB_CUDA(cudaStreamSynchronize(s));
}

void build_p2m_work_dev(fmmb_plan* pl, cudaStream_t s) {
  const int nleaf = pl->nbox_j[pl->lmax], per = kP2MItem;
  TmpBuf<int> cnt(s);
  cnt.alloc((size_t)nleaf + 1);
  FMMB_CUDA(cudaMemsetAsync(cnt.get() + nleaf, 0, sizeof(int), s));
  if (nleaf > 0) {
    src_item_counts<<<nblk(nleaf, kT), kT, 0, s>>>(nleaf, per, pl->leaf_j.get(), cnt.get());
    FMMB_CHECK_LAUNCH();
  }
  exclusive_scan(cnt.get(), nleaf + 1, s);
  const int n = d2h_int(cnt.get() + nleaf, s);
  pl->p2m_work.alloc(std::max(n, 1));
  pl->p2m_nwork = n;
  if (nleaf > 0) {
    src_items<<<nblk(nleaf, kT), kT, 0, s>>>(nleaf, per, pl->leaf_j.get(), cnt.get(), pl->p2m_work.get());
    FMMB_CHECK_LAUNCH();
  }
  FMMB_CUDA(cudaStreamSynchronize(s));
}

void build_inverse_perm_dev(fmmb_plan* pl, cudaStream_t s) {
  pl->inv_i.alloc(std::max(pl->ni, 1));
  if (pl->ni > 0) {
    invert_perm<<<nblk(pl->ni, kT), kT, 0, s>>>(pl->ni, pl->perm_i.get(), pl->inv_i.get());
    FMMB_CHECK_LAUNCH();
  }
}

}  // namespace fmmb
