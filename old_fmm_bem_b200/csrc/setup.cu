// Device-side construction of the evaluation work lists of a geometry
// (fmmb_set_geometry): the M2L pair tiles (tensor-core and FP64 forms) and the CSR
// of the tensor-core form's per-box reduction, the M2M / L2L tiles, the near-field
// work items, the inverse target permutation.  Scans and stable radix sorts
// (tree.cu) over the device lists the tree build produced, so that none of it is
// copied to the host.
//
// Bound: launches and the few read-backs (pair, tile and item counts) that
// allocations wait for; the lists themselves are a few passes over the box slots.
// Measured on one B200 against M2M / L2L tiles and tree checks on the host, a
// second sort for the CSR, one atomic per pair or box and a second tree build for
// a set that is both targets and sources, fmmb_set_geometry called with the same
// points again, so that no buffer of the plan grows: 131,071 clustered
// points 2.34 -> 1.00 ms, 1,048,576 13.3 -> 8.8 ms, 100,000 points in reference
// semantics from host arrays 2.68 -> 0.86 ms.
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

// first position of each key in the sorted list, for keys 0..nk (start[nk] = n)
__global__ void key_starts(int nk, int n, const int* __restrict__ key, int* __restrict__ start) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o > nk) return;
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (key[mid] < o) lo = mid + 1;
    else hi = mid;
  }
  start[o] = lo;
}

__global__ void tiles_per_key(int nk, int tt, const int* __restrict__ start, int* __restrict__ tiles) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o <= nk) tiles[o] = o < nk ? (start[o + 1] - start[o] + tt - 1) / tt : 0;
}

// sorted pair j -> tile tile_base[op] + r / tt, column r % tt (r = its rank
// among the pairs of its operator); col (may be null): the column of each pair
// in enumeration order, tile * tt + column
__global__ void fill_tiles(int n, int tt, const int* __restrict__ opk, const int* __restrict__ ord,
                           const int* __restrict__ src, const int* __restrict__ dst, const int* __restrict__ phi,
                           const int* __restrict__ op_start, const int* __restrict__ tile_base,
                           int* __restrict__ tile_op, int* __restrict__ tile_src, int* __restrict__ tdst,
                           int* __restrict__ tile_phi, int* __restrict__ col) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int op = opk[j], r = j - op_start[op];
  const int t = tile_base[op] + r / tt, c = r % tt;
  tile_src[(size_t)t * tt + c] = src[ord[j]];
  if (tdst) tdst[(size_t)t * tt + c] = dst[ord[j]];
  if (col) col[ord[j]] = t * tt + c;
  if (phi) tile_phi[(size_t)t * tt + c] = phi[ord[j]];
  if (c == 0) tile_op[t] = op;
}

__global__ void fill_tile_y(int ntile, int* __restrict__ ty) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntile) return;
  ty[2 * t] = t * 128;
  ty[2 * t + 1] = 0;
}

// row (target box) -> its pairs: the enumeration visits the boxes in order, so
// they are consecutive; ptr[row] from the scanned slot flags
__global__ void row_ptrs(int nrow, LevTab T, const int* __restrict__ pos, int npair, int* __restrict__ rows,
                         int* __restrict__ ptr) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r > nrow) return;
  if (r == nrow) {
    ptr[r] = npair;
    return;
  }
  // rows in enumeration order: level l's boxes are vstart[l] / 189 + ...
  int l = 0;
  while (l + 1 < T.nlev && T.vstart[l + 1] / kM2LSlots <= r) l++;
  rows[r] = T.boxoff[l] + r - T.vstart[l] / kM2LSlots;
  ptr[r] = pos[r * kM2LSlots];
}

// ---- M2M / L2L pair tiles: {operator, input row, output row} of every box of
// levels 3..lmax and its parent, grouped by level and child octant ----
struct PairTab {
  int lmax;
  int off[kMaxLev], tile0[kMaxLev];  // per level: first box in the all-level arrays (lmax first), first tile
  int op0[kMaxLev];                  // operator of octant 0 of the level's pairs
};
__device__ __forceinline__ int level_of(const PairTab& T, int c) {
  int lev = T.lmax;
  while (lev > 3 && c >= T.off[lev - 1]) lev--;
  return lev;
}
// rank of box c among the boxes of its (level, octant): one atomic per warp and group
__device__ __forceinline__ int group_rank(int g, int* cnt) {
  const unsigned peers = __match_any_sync(__activemask(), g);
  const int lane = threadIdx.x & 31, lead = __ffs(peers) - 1;
  int base = 0;
  if (lane == lead) base = atomicAdd(&cnt[g], __popc(peers));
  return __shfl_sync(peers, base, lead) + __popc(peers & ((1u << lane) - 1u));
}
__global__ void pair_counts(int n, PairTab T, const int* __restrict__ key, int* __restrict__ cnt) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < n) group_rank(8 * level_of(T, c) + (key[c] & 7), cnt);
}
// one block: first tile of each (level, octant), and the tiles' operators
__global__ void pair_bases(PairTab T, int tt, const int* __restrict__ cnt, int* __restrict__ base, int* __restrict__ tile_op) {
  for (int lev = 3; lev <= T.lmax; lev++) {
    int t = T.tile0[lev];
    for (int o = 0; o < 8; o++) {
      const int nt = (cnt[8 * lev + o] + tt - 1) / tt;
      if (threadIdx.x == 0) base[8 * lev + o] = t;
      for (int k = threadIdx.x; k < nt; k += blockDim.x) tile_op[t + k] = T.op0[lev] + o;
      t += nt;
    }
  }
}
// up: the parent is the output (M2M), else the input (L2L)
__global__ void pair_fill(int n, PairTab T, int tt, bool up, const int* __restrict__ key, const int* __restrict__ parent,
                          const int* __restrict__ base, int* __restrict__ cursor, int* __restrict__ tile_src,
                          int* __restrict__ tile_dst) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  const int lev = level_of(T, c), g = 8 * lev + (key[c] & 7);
  const size_t at = (size_t)base[g] * tt + group_rank(g, cursor);
  const int par = T.off[lev - 1] + parent[c];
  tile_src[at] = up ? c : par;
  tile_dst[at] = up ? par : c;
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

// one launch (n0 = n): in order; two: sorted item j -> launch (j & 1), position j >> 1 within it
__global__ void deal_items(int n, int n0, const int* __restrict__ sorted, const int2* __restrict__ work,
                           int2* __restrict__ out) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int o = n0 == n ? j : (j & 1) ? n0 + (j >> 1) : j >> 1;
  out[o] = work[sorted[j]];
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
// rel_to_op[r].  tile_dst / tile_phi (may be null): the target row and the azimuth
// index of each pair; csr (may be null): per target box its pairs' columns
// (tile * tt + column), in slot order.  False when the enumeration does not fit
// an int.
struct M2LTiles {
  int npair = 0, ntile = 0;
};
bool build_m2l_tiles(fmmb_plan* pl, bool sets, int per, const int* rel_to_op, int tt, DevBuf<int>& tile_op,
                     DevBuf<int>& tile_src, DevBuf<int>* tile_dst, DevBuf<int>* tile_phi, fmmb_plan::TcJob* csr,
                     M2LTiles& out, cudaStream_t s) {
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
    // the host loops take such sizes; the last blocks of the kernels and of the scan
    // (tiles of 4,096) index past V, which must not wrap around
    if (V >= (1LL << 31) - 8192) return false;
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
  const int npair = (int)pl->m2l_pairs;  // counted, and read back, with the tree
  if (csr) {
    const int nrow = nv / kM2LSlots;
    csr->nred = npair > 0 ? nrow : 0;
    csr->red_rows.alloc(std::max(nrow, 1));
    csr->red_ptr.alloc((size_t)nrow + 1);
    csr->red_idx.alloc(std::max(npair, 1));
    row_ptrs<<<nblk(nrow + 1, kT), kT, 0, s>>>(nrow, T, pos.get(), npair, csr->red_rows.get(), csr->red_ptr.get());
    FMMB_CHECK_LAUNCH();
  }
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
  TmpBuf<int> op_start(s), tile_base(s);
  op_start.alloc(nops + 1);
  tile_base.alloc(nops + 1);
  key_starts<<<nblk(nops + 1, kT), kT, 0, s>>>(nops, npair, opk.get(), op_start.get());
  FMMB_CHECK_LAUNCH();
  tiles_per_key<<<nblk(nops + 1, kT), kT, 0, s>>>(nops, tt, op_start.get(), tile_base.get());
  FMMB_CHECK_LAUNCH();
  exclusive_scan(tile_base.get(), nops + 1, s);
  const int ntile = d2h_int(tile_base.get() + nops, s);
  const size_t ncol = (size_t)std::max(ntile, 1) * tt;
  tile_op.alloc(std::max(ntile, 1));
  tile_src.alloc(ncol);
  FMMB_CUDA(cudaMemsetAsync(tile_src.get(), 0xff, ncol * sizeof(int), s));
  if (tile_dst) {
    tile_dst->alloc(ncol);
    FMMB_CUDA(cudaMemsetAsync(tile_dst->get(), 0xff, ncol * sizeof(int), s));
  }
  if (tile_phi) {
    tile_phi->alloc(ncol);
    FMMB_CUDA(cudaMemsetAsync(tile_phi->get(), 0, ncol * sizeof(int), s));
  }
  if (npair > 0) {
    fill_tiles<<<nblk(npair, kT), kT, 0, s>>>(npair, tt, opk.get(), ord.get(), src.get(), dst.get(),
                                             tile_phi ? phi.get() : nullptr, op_start.get(), tile_base.get(),
                                             tile_op.get(), tile_src.get(), tile_dst ? tile_dst->get() : nullptr,
                                             tile_phi ? tile_phi->get() : nullptr, csr ? csr->red_idx.get() : nullptr);
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
  if (build_m2l_tiles(pl, sets, ncls, pl->d_rel_to_cls.get(), 32, job.tile_op, job.tile_src, &job.tile_dst, &job.tile_phi,
                      nullptr, t, s)) {
    job.ntile = t.ntile;
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
}

// The tiles are placed by an upper bound of their number (a level's boxes / 32 +
// 8), so that nothing is read back: the few left over have operator -1 and no
// work.
void build_pair_jobs(fmmb_plan* pl, int m2m0, int l2l0, int ops_per_level, cudaStream_t s) {
  const int lmax = pl->lmax, tt = pairs_f64_tile();
  for (int up = 0; up < 2; up++) {
    const std::vector<int>& nbox = up ? pl->nbox_j : pl->nbox_i;
    const std::vector<int>& off = up ? pl->off_j : pl->off_i;
    fmmb_plan::PairTiles& job = up ? pl->m2m_tiles : pl->l2l_tiles;
    PairTab T{};
    T.lmax = lmax;
    job.first.assign(lmax + 1, 0);
    job.ntile.assign(lmax + 1, 0);
    int nt = 0;
    for (int lev = lmax; lev >= 2; lev--) {
      T.off[lev] = off[lev];
      T.tile0[lev] = nt;
      T.op0[lev] = (up ? m2m0 : l2l0) + (lev - 3) * ops_per_level;
      if (lev < 3) continue;
      job.first[lev] = nt;
      job.ntile[lev] = nbox[lev] / tt + 8;
      nt += job.ntile[lev];
    }
    const int n = lmax >= 3 ? off[2] : 0;  // boxes of levels 3..lmax
    const size_t ncol = (size_t)std::max(nt, 1) * tt;
    job.op.alloc(std::max(nt, 1));
    job.src.alloc(ncol);
    job.dst.alloc(ncol);
    if (n == 0) continue;
    FMMB_CUDA(cudaMemsetAsync(job.op.get(), 0xff, nt * sizeof(int), s));
    FMMB_CUDA(cudaMemsetAsync(job.src.get(), 0xff, ncol * sizeof(int), s));
    FMMB_CUDA(cudaMemsetAsync(job.dst.get(), 0xff, ncol * sizeof(int), s));
    TmpBuf<int> tab(s);  // counts, cursors, first tiles of each (level, octant)
    const int ng = 8 * (lmax + 1);
    tab.alloc(3 * ng);
    FMMB_CUDA(cudaMemsetAsync(tab.get(), 0, 3 * ng * sizeof(int), s));
    const int* key = (up ? pl->key_j : pl->key_i).get();
    const int* parent = (up ? pl->parent_j : pl->parent_i).get();
    pair_counts<<<nblk(n, kT), kT, 0, s>>>(n, T, key, tab.get());
    FMMB_CHECK_LAUNCH();
    pair_bases<<<1, kT, 0, s>>>(T, tt, tab.get(), tab.get() + 2 * ng, job.op.get());
    FMMB_CHECK_LAUNCH();
    pair_fill<<<nblk(n, kT), kT, 0, s>>>(n, T, tt, up == 1, key, parent, tab.get() + 2 * ng, tab.get() + ng,
                                         job.src.get(), job.dst.get());
    FMMB_CHECK_LAUNCH();
  }
}

bool build_m2l_job_dev(fmmb_plan* pl, fmmb_plan::TcJob& job, int ys, cudaStream_t s) {
  M2LTiles t;
  if (!build_m2l_tiles(pl, pl->ops.m2l_sets > 1, 316, pl->d_rel_to_op.get(), 128, job.tile_op, job.tile_src, nullptr,
                       nullptr, &job, t, s))
    return false;
  const int ntile = t.ntile;
  job.ntile = ntile;
  job.tile_y.alloc((size_t)std::max(ntile, 1) * 2);
  if (ntile > 0) {
    fill_tile_y<<<nblk(ntile, kT), kT, 0, s>>>(ntile, job.tile_y.get());
    FMMB_CHECK_LAUNCH();
  }
  job.ys = ys;
  pl->tc_y.alloc((size_t)std::max(ntile, 1) * 128 * ys);
  return true;
}

void build_work_dev(fmmb_plan* pl, bool tc_m2l, cudaStream_t s) {
  const int nleaf = pl->nbox_i[pl->lmax], nleaf_j = pl->nbox_j[pl->lmax], per = kP2MItem;
  TmpBuf<int> cnt(s), cnt_j(s);
  TmpBuf<long long> nsrc(s);
  cnt.alloc((size_t)nleaf + 1);
  cnt_j.alloc((size_t)nleaf_j + 1);
  nsrc.alloc(std::max(nleaf, 1));
  FMMB_CUDA(cudaMemsetAsync(cnt.get() + nleaf, 0, sizeof(int), s));
  FMMB_CUDA(cudaMemsetAsync(cnt_j.get() + nleaf_j, 0, sizeof(int), s));
  if (nleaf > 0) {
    leaf_item_counts<<<nblk(nleaf, kT), kT, 0, s>>>(nleaf, pl->leaf_i.get(), pl->leaf_j.get(), pl->p2p_list.get(),
                                                   cnt.get(), nsrc.get());
    FMMB_CHECK_LAUNCH();
  }
  if (nleaf_j > 0) {
    src_item_counts<<<nblk(nleaf_j, kT), kT, 0, s>>>(nleaf_j, per, pl->leaf_j.get(), cnt_j.get());
    FMMB_CHECK_LAUNCH();
  }
  exclusive_scan(cnt.get(), nleaf + 1, s);
  exclusive_scan(cnt_j.get(), nleaf_j + 1, s);
  int tot[2];
  FMMB_CUDA(cudaMemcpyAsync(&tot[0], cnt.get() + nleaf, sizeof(int), cudaMemcpyDeviceToHost, s));
  FMMB_CUDA(cudaMemcpyAsync(&tot[1], cnt_j.get() + nleaf_j, sizeof(int), cudaMemcpyDeviceToHost, s));
  FMMB_CUDA(cudaStreamSynchronize(s));
  const int n = tot[0];
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
  // One launch of the near field, beside the far field from its start on; two
  // halves, before and after the M2L, where the tensor-core M2L, which takes whole
  // SMs, would have to wait for a long first one.  Both sides measured, two against
  // one (repeats differ by 0.2 %), at 2,744 to 3,375 items (p = 8 to 12, 24 or 64
  // points a leaf) between 3 % less and 1.6 % more, 2,989 items launched directly
  // (131,071 points moved and evaluated) 1,072 / 1,055 us; from 4,096 on never more
  // than 0.5 % more: 4,096 items 493 / 511 us at p = 12, 595 / 593 at p = 10, 4,626
  // (245,760 points on a surface) 350 / 356, 10,648 at p = 12 1,147 / 1,177, 21,892
  // (1,048,576 clustered points, forward and backward) 9.69 / 9.74 ms, 32,768 and
  // more between 1.4 % less and equal.  Without a tensor-core M2L one is better
  // throughout (32,768 points FP64, 512 items, 257 -> 173 us; 262,144 clustered
  // points 2.60 -> 2.43 ms).
  const int n0 = tc_m2l && n >= (1 << 12) ? (n + 1) / 2 : n;
  pl->p2p_work.alloc(std::max(n, 1));
  if (n > 0) {
    deal_items<<<nblk(n, kT), kT, 0, s>>>(n, n0, sval.get(), pl->m_p2p_work.get(), pl->p2p_work.get());
    FMMB_CHECK_LAUNCH();
  }
  pl->p2p_nwork = n;
  pl->p2p_nwork0 = n0;
  pl->p2m_work.alloc(std::max(tot[1], 1));
  pl->p2m_nwork = tot[1];
  if (nleaf_j > 0) {
    src_items<<<nblk(nleaf_j, kT), kT, 0, s>>>(nleaf_j, per, pl->leaf_j.get(), cnt_j.get(), pl->p2m_work.get());
    FMMB_CHECK_LAUNCH();
  }
}

void build_inverse_perm_dev(fmmb_plan* pl, cudaStream_t s) {
  pl->inv_i.alloc(std::max(pl->ni, 1));
  if (pl->ni > 0) {
    invert_perm<<<nblk(pl->ni, kT), kT, 0, s>>>(pl->ni, pl->perm_i.get(), pl->inv_i.get());
    FMMB_CHECK_LAUNCH();
  }
}

}  // namespace fmmb
