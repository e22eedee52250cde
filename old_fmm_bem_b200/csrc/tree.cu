// Octree construction on the GPU.
//
// Replaces the reference's serial tree build: box keys (fmm/boxn.cxx:5-31),
// the stable counting sort and the particle permutation (sort/csort.cxx:5-17,
// sort/sorti.cxx:12-35, sort/sortj.cxx:12-36), leaf ranges
// (fmm/boxdatai.cxx:10-34, fmm/boxdataj.cxx:10-36), parent levels
// (fmm/boxm2mi.cxx:6-24, fmm/boxm2mj.cxx:6-26) and the neighbour and
// interaction lists (fmm/ijbox.cxx:9-117).  The result is bit-identical to the
// reference: same keys (same float/double rounding), same stable order, same
// list entries in the same order.
//
// Lists are stored densely: 27 slots per target leaf for the near field and
// 189 slots per target box for M2L, -1 where the source box is empty.  The
// slot order is the reference's loop order, so dropping the -1 entries gives
// the reference lists.
//
// Forest (many independent problems in one plan): the problem index of a
// point sits above its 3*lmax Morton bits, so the sort groups the points by
// problem, every box belongs to one problem (its key at level l is
// (problem << 3l) | morton), and a neighbour or interaction-list lookup only
// finds boxes of the same problem.  With one problem the keys are the
// reference's.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cstring>
#include <mutex>

#include "internal.h"

namespace fmmb {

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;

// exclusive prefix of v over the block's threads; total: the block's sum
__device__ __forceinline__ int block_prefix(int v, int& total) {
  __shared__ int ws[kScanThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  __syncthreads();  // the previous use of ws is over
  if (lane == 31) ws[w] = incl;
  __syncthreads();
  int before = 0;
  total = 0;
#pragma unroll
  for (int k = 0; k < kScanThreads / 32; k++) {
    if (k < w) before += ws[k];
    total += ws[k];
  }
  return before + incl - v;
}

// sum of each tile
__global__ void __launch_bounds__(kScanThreads) scan_sums(const int* __restrict__ data, int n, int* __restrict__ sums) {
  const int base = blockIdx.x * kScanTile;
  int t = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; i++) {
    const int j = base + i * kScanThreads + threadIdx.x;
    t += j < n ? data[j] : 0;
  }
  int total;
  block_prefix(t, total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// exclusive scan of each tile, from the sum of the tiles before it (`sums`:
// their sums, or, PREFIX, already their exclusive scan; null: one tile)
template <bool PREFIX>
__global__ void __launch_bounds__(kScanThreads) scan_tiles(int* __restrict__ data, int n, const int* __restrict__ sums) {
  int off = 0;
  if (sums) {
    if (PREFIX) {
      off = sums[blockIdx.x];
    } else {
      int t = 0;
      for (int k = threadIdx.x; k < (int)blockIdx.x; k += kScanThreads) t += sums[k];
      block_prefix(t, off);
    }
  }
  // a warp's items are consecutive: 16 rows of 32
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int base = blockIdx.x * kScanTile + w * 32 * kScanItems;
  int v[kScanItems], t = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; i++) {
    const int j = base + i * 32 + lane;
    v[i] = j < n ? data[j] : 0;
    t += v[i];
  }
  int wsum = t;
#pragma unroll
  for (int o = 16; o; o >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
  int total;
  const int before = block_prefix(lane == 0 ? wsum : 0, total);
  int run = off + __shfl_sync(0xffffffffu, before, 0);
#pragma unroll
  for (int i = 0; i < kScanItems; i++) {
    const int j = base + i * 32 + lane;
    int incl = v[i];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
    }
    if (j < n) data[j] = run + incl - v[i];
    run += __shfl_sync(0xffffffffu, incl, 31);
  }
}

}  // namespace

// In-place exclusive scan: the tiles' sums, then every tile on top of the sums
// before it, which its block adds up itself (two launches; three tile-local
// passes before).  Above 4,096 tiles (16.8 M items) the sums are scanned first:
// adding them up per block would read more than the data.
void exclusive_scan(int* data, int n, cudaStream_t s) {
  if (n <= 0) return;
  const int nb = (n + kScanTile - 1) / kScanTile;
  if (nb == 1) {
    scan_tiles<false><<<1, kScanThreads, 0, s>>>(data, n, nullptr);
    FMMB_CHECK_LAUNCH();
    return;
  }
  TmpBuf<int> sums(s);  // freed in stream order
  sums.alloc(nb);
  scan_sums<<<nb, kScanThreads, 0, s>>>(data, n, sums.get());
  FMMB_CHECK_LAUNCH();
  if (nb <= 4096) {
    scan_tiles<false><<<nb, kScanThreads, 0, s>>>(data, n, sums.get());
  } else {
    exclusive_scan(sums.get(), nb, s);
    scan_tiles<true><<<nb, kScanThreads, 0, s>>>(data, n, sums.get());
  }
  FMMB_CHECK_LAUNCH();
}

cudaMemPool_t scratch_pool() {
  static std::mutex mu;
  static cudaMemPool_t pools[64] = {};
  int dev = 0;
  FMMB_CUDA(cudaGetDevice(&dev));
  FMMB_REQUIRE(dev >= 0 && dev < 64, FMMB_ERR_ARG, "device ordinal out of range");
  std::lock_guard<std::mutex> lk(mu);
  if (!pools[dev]) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    FMMB_CUDA(cudaMemPoolCreate(&pool, &props));
    uint64_t keep = kScratchPoolKeep;
    FMMB_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    pools[dev] = pool;
  }
  return pools[dev];
}

namespace {

// ---- stable LSD radix sort of (key, index) ----
constexpr int kRsWarps = 8;
constexpr int kRsThreads = kRsWarps * 32;
// Elements per thread (ROUNDS): 8, and 2 below 2^18 elements, where blocks of 2,048
// are fewer than the 148 SMs.  fmmb_set_geometry with 8 / 2: 65,536 points 0.631 /
// 0.560 ms, 131,072 0.609 / 0.565; 262,144 1.026 / 1.037, 393,216 1.033 / 1.054,
// 1,048,576 1.132 / 1.141.
template <int ROUNDS>
__global__ void rs_hist(const int* keys, int n, int shift, int nblocks, int* counts) {
  constexpr int kRsTile = kRsThreads * ROUNDS;
  __shared__ int h[256];
  for (int d = threadIdx.x; d < 256; d += blockDim.x) h[d] = 0;
  __syncthreads();
  const int base = blockIdx.x * kRsTile;
  for (int i = threadIdx.x; i < kRsTile; i += blockDim.x)
    if (base + i < n) atomicAdd(&h[(keys[base + i] >> shift) & 255], 1);
  __syncthreads();
  for (int d = threadIdx.x; d < 256; d += blockDim.x) counts[d * nblocks + blockIdx.x] = h[d];
}

// Each warp owns a contiguous run of ROUNDS*32 elements, processed 32 at a
// time in order; ranks among equal digits come from __match_any_sync, so the
// scatter keeps the input order of equal keys (stable).
template <int kRsRounds>
__global__ void rs_scatter(const int* kin, const int* vin, int* kout, int* vout, int n, int shift, int nblocks,
                           const int* offsets) {
  constexpr int kRsTile = kRsThreads * kRsRounds;
  __shared__ int wc[kRsWarps][256];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int d = threadIdx.x; d < 256 * kRsWarps; d += blockDim.x) (&wc[0][0])[d] = 0;
  __syncthreads();
  const int base = blockIdx.x * kRsTile + w * (kRsRounds * 32);
  const unsigned lt = (1u << lane) - 1;
  int rank[kRsRounds], dig[kRsRounds], key[kRsRounds], val[kRsRounds];
#pragma unroll
  for (int r = 0; r < kRsRounds; r++) {
    const int i = base + r * 32 + lane;
    const bool ok = i < n;
    key[r] = ok ? kin[i] : 0;
    val[r] = ok ? vin[i] : 0;
    const int d = ok ? ((key[r] >> shift) & 255) : (256 + lane);
    dig[r] = d;
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    const int before = __popc(peers & lt);
    const int prior = ok ? wc[w][d] : 0;
    __syncwarp();
    if (ok && before == 0) wc[w][d] = prior + __popc(peers);
    __syncwarp();
    rank[r] = prior + before;
  }
  __syncthreads();
  if (threadIdx.x < 256) {
    int run = 0;
    for (int ww = 0; ww < kRsWarps; ww++) {
      int t = wc[ww][threadIdx.x];
      wc[ww][threadIdx.x] = run;
      run += t;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kRsRounds; r++) {
    const int d = dig[r];
    if (d < 256) {
      const int pos = offsets[d * nblocks + blockIdx.x] + wc[w][d] + rank[r];
      kout[pos] = key[r];
      vout[pos] = val[r];
    }
  }
}

}  // namespace

void radix_sort(int* keys, int* vals, int n, int bits, cudaStream_t s) {
  if (n <= 1 || bits <= 0) return;
  const bool small = n < (1 << 18);
  const int tile = kRsThreads * (small ? 2 : 8), nb = (n + tile - 1) / tile;
  TmpBuf<int> k2(s), v2(s), counts(s);
  k2.alloc(n);
  v2.alloc(n);
  counts.alloc((size_t)256 * nb);
  int *ka = keys, *va = vals, *kb = k2.get(), *vb = v2.get();
  int passes = 0;
  for (int shift = 0; shift < bits; shift += 8, passes++) {
    (small ? rs_hist<2> : rs_hist<8>)<<<nb, kRsThreads, 0, s>>>(ka, n, shift, nb, counts.get());
    FMMB_CHECK_LAUNCH();
    exclusive_scan(counts.get(), 256 * nb, s);
    (small ? rs_scatter<2> : rs_scatter<8>)<<<nb, kRsThreads, 0, s>>>(ka, va, kb, vb, n, shift, nb, counts.get());
    FMMB_CHECK_LAUNCH();
    std::swap(ka, kb);
    std::swap(va, vb);
  }
  if (passes & 1) {
    FMMB_CUDA(cudaMemcpyAsync(keys, ka, n * sizeof(int), cudaMemcpyDeviceToDevice, s));
    FMMB_CUDA(cudaMemcpyAsync(vals, va, n * sizeof(int), cudaMemcpyDeviceToDevice, s));
  }
}

namespace {

// ---- keys (fmm/boxn.cxx:5-31) ----
__device__ __forceinline__ int morton(int cx, int cy, int cz, int lev) {
  int k = 0;
  for (int i = 0; i < lev; i++)
    k |= (((cx >> i) & 1) << (3 * i + 1)) | (((cy >> i) & 1) << (3 * i)) | (((cz >> i) & 1) << (3 * i + 2));
  return k;
}
__device__ __forceinline__ void demorton(int k, int& cx, int& cy, int& cz) {
  cx = cy = cz = 0;
  for (int i = 0; i < 10; i++) {
    cy |= ((k >> (3 * i)) & 1) << i;
    cx |= ((k >> (3 * i + 1)) & 1) << i;
    cz |= ((k >> (3 * i + 2)) & 1) << i;
  }
}

// The reference truncates (x - xmin) [float] * rb [double, from the float
// division kl/rd] and moves the last boundary back by one box.  Points below
// the root corner are clamped to box 0 (the reference leaves them undefined).
__device__ __forceinline__ int box_coord(float x, float xmin, double rb, int kl) {
  const float d = __fsub_rn(x, xmin);
  int c = (int)__dmul_rn((double)d, rb);
  if (c >= kl) c--;
  if (c >= kl) c = kl - 1;
  if (c < 0) c = 0;
  return c;
}

// off[0..nprob]: first point of each problem (off[nprob] = n)
__global__ void keys_kernel(int n, const float* x, const float* y, const float* z, float xmin, float ymin, float zmin,
                            double rb, int lmax, int nprob, const int* off, int* key, int* idx) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int kl = 1 << lmax;
  int pid = 0;
  if (nprob > 1) {  // last problem whose first point is <= i
    int lo = 0, hi = nprob - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (off[mid] <= i) lo = mid;
      else hi = mid - 1;
    }
    pid = lo;
  }
  key[i] = (pid << (3 * lmax)) |
           morton(box_coord(x[i], xmin, rb, kl), box_coord(y[i], ymin, rb, kl), box_coord(z[i], zmin, rb, kl), lmax);
  idx[i] = i;
}

// spatial part of the keys (problem bits removed)
__global__ void mask_keys(int n, const int* key, int mask, int* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = key[i] & mask;
}

__global__ void gather_points(int n, const int* perm, const float* x, const float* y, const float* z, const float* nx,
                              const float* ny, const float* nz, float4* pos, float4* nrm) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int o = perm[i];
  pos[i] = make_float4(x[o], y[o], z[o], 0.f);
  nrm[i] = nx ? make_float4(nx[o], ny[o], nz[o], 0.f) : make_float4(0.f, 0.f, 0.f, 0.f);
}

// flag[i] = 1 where a new run of (key >> shift) starts
__global__ void run_flags(int n, const int* key, int shift, int* flag, int* flag_copy) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int f = (i == 0 || (key[i] >> shift) != (key[i - 1] >> shift)) ? 1 : 0;
  flag[i] = f;
  flag_copy[i] = f;
}

// runs of a level = last scanned flag + last flag
__global__ void run_count(int n, const int* scanned, const int* flag_copy, int* count) {
  *count = n > 0 ? scanned[n - 1] + flag_copy[n - 1] : 0;
}

// After the exclusive scan of the flags: write compact keys, run starts and
// the run index of every element.
__global__ void run_compact(int n, const int* key, int shift, const int* scanned, const int* flag_copy, int* out_key,
                            int* out_first, int* elem_run) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int r = scanned[i] + flag_copy[i] - 1;
  if (elem_run) elem_run[i] = r;
  if (flag_copy[i]) {
    out_key[r] = key[i] >> shift;
    if (out_first) out_first[r] = i;
  }
}

__global__ void leaf_ranges(int nleaf, int n, const int* first, int2* leaf) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nleaf) return;
  const int f = first[b];
  const int e = (b + 1 < nleaf) ? first[b + 1] : n;
  leaf[b] = make_int2(f, e - f);
}

// A broken tree must not reach the expansion kernels: the parents of a level's
// boxes start at 0, grow by 0 or 1, end at nparent - 1 and none has more than 8
// children.
__global__ void check_parents(int nchild, const int* __restrict__ parent, int nparent, int* __restrict__ bad) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nchild) return;
  const int p = parent[c], before = c ? parent[c - 1] : -1;
  const bool ok = p >= 0 && p < nparent && (c == 0 ? p == 0 : (p == before || p == before + 1)) &&
                  (c < nchild - 1 || p == nparent - 1) && (c < 8 || parent[c - 8] != p);
  if (!ok) *bad = 1;
}

__device__ __forceinline__ int find_key(const int* keys, int n, int k) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (keys[mid] < k) lo = mid + 1;
    else hi = mid;
  }
  return (lo < n && keys[lo] == k) ? lo : -1;
}

// Near-field slots (fmm/ijbox.cxx:30-53): jx, jy, jz ascending over the 3x3x3
// neighbourhood, self included; one thread per slot.
__global__ void p2p_lists(int nleaf_i, const int* key_i, int nleaf_j, const int* key_j, int lev, int* list) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= (long long)nleaf_i * kP2PSlots) return;
  const int b = (int)(t / kP2PSlots), s = (int)(t % kP2PSlots);
  int ix, iy, iz;
  const int smask = (1 << (3 * lev)) - 1, prob = key_i[b] & ~smask;
  demorton(key_i[b] & smask, ix, iy, iz);
  const int kl = 1 << lev;
  const int jx = ix + s / 9 - 1, jy = iy + (s / 3) % 3 - 1, jz = iz + s % 3 - 1;
  int v = -1;
  if (jx >= 0 && jx < kl && jy >= 0 && jy < kl && jz >= 0 && jz < kl)
    v = find_key(key_j, nleaf_j, prob | morton(jx, jy, jz, lev));
  list[t] = v;
}

// Interaction-list slots (fmm/ijbox.cxx:74-109), relative offsets per octant
// from slot_rel.
__global__ void m2l_lists(int nbox_i, const int* key_i, int nbox_j, const int* key_j, int lev, const int* slot_rel,
                          int* list) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nbox_i * kM2LSlots) return;
  const int b = t / kM2LSlots, s = t % kM2LSlots;
  const int key = key_i[b];
  const int smask = (1 << (3 * lev)) - 1, prob = key & ~smask;
  int ix, iy, iz;
  demorton(key & smask, ix, iy, iz);
  const int code = slot_rel[(key & 7) * kM2LSlots + s];
  const int jx = ix - (code / 49 - 3), jy = iy - ((code / 7) % 7 - 3), jz = iz - (code % 7 - 3);
  const int kl = 1 << lev;
  int v = -1;
  if (jx >= 0 && jx < kl && jy >= 0 && jy < kl && jz >= 0 && jz < kl)
    v = find_key(key_j, nbox_j, prob | morton(jx, jy, jz, lev));
  list[t] = v;
}

// adds v over the block's threads to *out with one atomic
__device__ __forceinline__ void block_add(unsigned long long v, unsigned long long* out) {
  __shared__ unsigned long long ws[32];
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < (int)blockDim.x / 32; k++) v += ws[k];
    if (v) atomicAdd(out, v);
  }
}

__global__ void count_p2p_pairs(int nleaf_i, const int2* leaf_i, const int2* leaf_j, const int* list,
                                unsigned long long* out) {
  unsigned long long acc = 0;
  const size_t n = (size_t)nleaf_i * kP2PSlots;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    const int j = list[t];
    if (j >= 0) acc += (unsigned long long)leaf_i[t / kP2PSlots].y * (unsigned long long)leaf_j[j].y;
  }
  block_add(acc, out);
}

__global__ void count_nonneg(size_t n, const int* list, unsigned long long* out) {
  unsigned long long acc = 0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    acc += list[i] >= 0;
  block_add(acc, out);
}

__global__ void minmax_kernel(int n, const float* x, float* out /*[2] min,max*/) {
  float lo = FLT_MAX, hi = -FLT_MAX;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    lo = fminf(lo, x[i]);
    hi = fmaxf(hi, x[i]);
  }
  for (int o = 16; o; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if ((threadIdx.x & 31) == 0) {
    // order-preserving int encoding for atomics on floats
    int ilo = __float_as_int(lo), ihi = __float_as_int(hi);
    ilo = ilo >= 0 ? ilo : ilo ^ 0x7fffffff;
    ihi = ihi >= 0 ? ihi : ihi ^ 0x7fffffff;
    atomicMin((int*)&out[0], ilo);
    atomicMax((int*)&out[1], ihi);
  }
}

inline int blocks(size_t n, int t) { return (int)((n + t - 1) / t); }

__global__ void gather_int(int n, const int* idx, const int* src, int* dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = src[idx[i]];
}

struct Side {
  const float *x, *y, *z, *nx, *ny, *nz;
  int n;
  const int* off;  // device [nprob + 1] first point of each problem
};

int prob_bits(int nprob) {
  int b = 0;
  while ((1 << b) < nprob) b++;
  return b;
}

// Builds keys, order, sorted points and all levels of one point set.
// bad: device flag, set when the levels do not fit together.
void build_side(fmmb_plan* pl, const Side& sd, bool is_target, int* bad, cudaStream_t s) {
  const int n = sd.n, lmax = pl->lmax;
  TmpBuf<int> key(s), idx(s), flag(s), flag2(s), nbd(s);
  key.alloc(n);
  idx.alloc(n);
  const double rb = (double)((float)(1 << lmax) / pl->bbox[3]);  // kl/rd: float division, as the reference
  keys_kernel<<<blocks(n, 256), 256, 0, s>>>(n, sd.x, sd.y, sd.z, pl->bbox[0], pl->bbox[1], pl->bbox[2], rb, lmax,
                                              pl->nprob, sd.off, key.get(), idx.get());
  FMMB_CHECK_LAUNCH();
  radix_sort(key.get(), idx.get(), n, 3 * lmax + prob_bits(pl->nprob), s);
  DevBuf<int>& perm = is_target ? pl->perm_i : pl->perm_j;
  DevBuf<float4>& pos = is_target ? pl->tpos : pl->spos;
  DevBuf<float4>& nrm = is_target ? pl->tnrm : pl->snrm;
  perm.alloc(n);
  pos.alloc(n);
  nrm.alloc(n);
  FMMB_CUDA(cudaMemcpyAsync(perm.get(), idx.get(), n * sizeof(int), cudaMemcpyDeviceToDevice, s));
  gather_points<<<blocks(n, 256), 256, 0, s>>>(n, idx.get(), sd.x, sd.y, sd.z, sd.nx, sd.ny, sd.nz, pos.get(), nrm.get());
  FMMB_CHECK_LAUNCH();

  // Levels lmax..2: runs of key >> 3(lmax-lev) over the sorted points.  Level
  // lmax's runs are the leaves; parents come from the run index of the
  // first point of each child.
  std::vector<int>& nbox = is_target ? pl->nbox_i : pl->nbox_j;
  nbox.assign(lmax + 1, 0);
  // every level's runs at once (arrays of n, the bound), the counts read
  // back with one synchronisation
  std::vector<TmpBuf<int>> kstore, fstore, rstore;
  for (int lev = 0; lev <= lmax; lev++) {
    kstore.emplace_back(s);
    fstore.emplace_back(s);
    rstore.emplace_back(s);
  }
  flag.alloc(n);
  flag2.alloc(n);
  nbd.alloc(lmax + 1);
  for (int lev = lmax; lev >= 2; lev--) {
    const int shift = 3 * (lmax - lev);
    if (n > 0) {
      run_flags<<<blocks(n, 256), 256, 0, s>>>(n, key.get(), shift, flag.get(), flag2.get());
      FMMB_CHECK_LAUNCH();
    }
    exclusive_scan(flag.get(), n, s);
    run_count<<<1, 1, 0, s>>>(n, flag.get(), flag2.get(), nbd.get() + lev);
    FMMB_CHECK_LAUNCH();
    kstore[lev].alloc(n);
    fstore[lev].alloc(n);
    rstore[lev].alloc(n);
    if (n > 0) {
      run_compact<<<blocks(n, 256), 256, 0, s>>>(n, key.get(), shift, flag.get(), flag2.get(), kstore[lev].get(),
                                                 fstore[lev].get(), rstore[lev].get());
      FMMB_CHECK_LAUNCH();
    }
  }
  FMMB_CUDA(cudaMemcpyAsync(nbox.data(), nbd.get(), (lmax + 1) * sizeof(int), cudaMemcpyDeviceToHost, s));
  FMMB_CUDA(cudaStreamSynchronize(s));
  nbox[0] = nbox[1] = 0;
  // concatenated per-level arrays, lmax first (the reference's nlbi/nlbj layout)
  std::vector<int>& off = is_target ? pl->off_i : pl->off_j;
  off.assign(lmax + 1, 0);
  int tot = 0;
  for (int lev = lmax; lev >= 2; lev--) {
    off[lev] = tot;
    tot += nbox[lev];
  }
  (is_target ? pl->tot_i : pl->tot_j) = tot;
  DevBuf<int>& keys_all = is_target ? pl->key_i : pl->key_j;
  DevBuf<int>& parent_all = is_target ? pl->parent_i : pl->parent_j;
  keys_all.alloc(tot);
  parent_all.alloc(tot);
  FMMB_CUDA(cudaMemsetAsync(parent_all.get(), 0xff, tot * sizeof(int), s));
  for (int lev = lmax; lev >= 2; lev--) {
    FMMB_CUDA(cudaMemcpyAsync(keys_all.get() + off[lev], kstore[lev].get(), nbox[lev] * sizeof(int),
                              cudaMemcpyDeviceToDevice, s));
    if (lev > 2) {
      // parent of box b at lev = run index (at lev-1) of its first point
      const int nb = nbox[lev];
      gather_int<<<blocks(nb, 256), 256, 0, s>>>(nb, fstore[lev].get(), rstore[lev - 1].get(),
                                                 parent_all.get() + off[lev]);
      FMMB_CHECK_LAUNCH();
    }
  }
  // leaves
  DevBuf<int2>& leaf = is_target ? pl->leaf_i : pl->leaf_j;
  leaf.alloc(nbox[lmax]);
  leaf_ranges<<<blocks(nbox[lmax], 256), 256, 0, s>>>(nbox[lmax], n, fstore[lmax].get(), leaf.get());
  FMMB_CHECK_LAUNCH();
  // leaf keys without the problem bits (box centres of P2M / L2P)
  DevBuf<int>& lk = is_target ? pl->leafkey_i : pl->leafkey_j;
  lk.alloc(nbox[lmax]);
  mask_keys<<<blocks(nbox[lmax], 256), 256, 0, s>>>(nbox[lmax], keys_all.get() + off[lmax], (1 << (3 * lmax)) - 1,
                                                    lk.get());
  FMMB_CHECK_LAUNCH();
  for (int lev = lmax; lev >= 3; lev--) {
    check_parents<<<blocks(nbox[lev], 256), 256, 0, s>>>(nbox[lev], parent_all.get() + off[lev], nbox[lev - 1], bad);
    FMMB_CHECK_LAUNCH();
  }
}

// The sources' tree where they are the targets' points, given as the same
// arrays: a copy of the targets' (the normals may differ).
void copy_side(fmmb_plan* pl, const Side& sd, cudaStream_t s) {
  const int n = sd.n, lmax = pl->lmax;
  pl->nbox_j = pl->nbox_i;
  pl->off_j = pl->off_i;
  pl->tot_j = pl->tot_i;
  auto copy = [&](auto& to, const auto& from, size_t cnt) {
    to.alloc(cnt);
    FMMB_CUDA(cudaMemcpyAsync(to.get(), from.get(), cnt * sizeof(*to.get()), cudaMemcpyDeviceToDevice, s));
  };
  copy(pl->perm_j, pl->perm_i, n);
  copy(pl->key_j, pl->key_i, pl->tot_i);
  copy(pl->parent_j, pl->parent_i, pl->tot_i);
  copy(pl->leaf_j, pl->leaf_i, pl->nbox_i[lmax]);
  copy(pl->leafkey_j, pl->leafkey_i, pl->nbox_i[lmax]);
  pl->spos.alloc(n);
  pl->snrm.alloc(n);
  gather_points<<<blocks(n, 256), 256, 0, s>>>(n, pl->perm_j.get(), sd.x, sd.y, sd.z, sd.nx, sd.ny, sd.nz,
                                               pl->spos.get(), pl->snrm.get());
  FMMB_CHECK_LAUNCH();
}

}  // namespace

void build_tree(fmmb_plan* pl, int ni, const float* tx, const float* ty, const float* tz, const float* tnx,
                const float* tny, const float* tnz, int nj, const float* sx, const float* sy, const float* sz,
                const float* snx, const float* sny, const float* snz, const float* bbox_in) {
  cudaStream_t s = pl->st.main;
  FMMB_REQUIRE(3 * pl->cfg.lmax + prob_bits(pl->nprob) <= 30, FMMB_ERR_CAPACITY,
               "box keys: 3*lmax + ceil(log2(problems)) must stay within 30 bits");
  pl->ni = ni;
  pl->nj = nj;
  pl->lmax = pl->cfg.lmax;
  if (bbox_in) {
    for (int k = 0; k < 4; k++) pl->bbox[k] = bbox_in[k];
  } else {
    // root cube from the extent of all points, as the BEM drivers do
    // (biobem/fmm_matmult.h:29-114): corner at the minimum, side = largest
    // extent * (1 + 1e-5).
    TmpBuf<float> mm(s);
    mm.alloc(6 * 2);
    float init[12];
    for (int k = 0; k < 6; k++) {
      init[2 * k] = FLT_MAX;
      init[2 * k + 1] = -FLT_MAX;
    }
    // encode initial values like minmax_kernel does
    int enc[12];
    for (int k = 0; k < 12; k++) {
      int v;
      std::memcpy(&v, &init[k], 4);
      enc[k] = v >= 0 ? v : v ^ 0x7fffffff;
    }
    FMMB_CUDA(cudaMemcpyAsync(mm.get(), enc, sizeof(enc), cudaMemcpyHostToDevice, s));
    const float* arr[6] = {tx, ty, tz, sx, sy, sz};
    for (int k = 0; k < 6; k++) {
      int n = k < 3 ? ni : nj;
      if (n > 0) minmax_kernel<<<std::min(blocks(n, 256), 1024), 256, 0, s>>>(n, arr[k], mm.get() + 2 * k);
      FMMB_CHECK_LAUNCH();
    }
    int res[12];
    FMMB_CUDA(cudaMemcpyAsync(res, mm.get(), sizeof(res), cudaMemcpyDeviceToHost, s));
    FMMB_CUDA(cudaStreamSynchronize(s));
    float v[12];
    for (int k = 0; k < 12; k++) {
      int e = res[k] >= 0 ? res[k] : res[k] ^ 0x7fffffff;
      std::memcpy(&v[k], &e, 4);
    }
    float lo[3], hi[3];
    for (int d = 0; d < 3; d++) {
      lo[d] = std::min(ni ? v[2 * d] : FLT_MAX, nj ? v[6 + 2 * d] : FLT_MAX);
      hi[d] = std::max(ni ? v[2 * d + 1] : -FLT_MAX, nj ? v[6 + 2 * d + 1] : -FLT_MAX);
    }
    float rd = 0;
    for (int d = 0; d < 3; d++) rd = std::max(rd, (hi[d] - lo[d]) * (1 + 1e-5f));
    if (!(rd > 0)) rd = 1;
    pl->bbox[0] = lo[0];
    pl->bbox[1] = lo[1];
    pl->bbox[2] = lo[2];
    pl->bbox[3] = rd;
  }
  FMMB_REQUIRE(pl->bbox[3] > 0, FMMB_ERR_ARG, "root box side must be positive");
  TmpBuf<unsigned long long> cnt(s);  // near-field pairs, M2L pairs, the tree check's flag
  cnt.alloc(3);
  FMMB_CUDA(cudaMemsetAsync(cnt.get(), 0, 3 * sizeof(unsigned long long), s));
  int* bad = reinterpret_cast<int*>(cnt.get() + 2);
  build_side(pl, Side{tx, ty, tz, tnx, tny, tnz, ni, pl->d_prob_off.get()}, true, bad, s);
  const Side src{sx, sy, sz, snx, sny, snz, nj, pl->d_prob_off.get() + pl->nprob + 1};
  if (pl->same_tree) copy_side(pl, src, s);
  else build_side(pl, src, false, bad, s);

  const int lmax = pl->lmax;
  const int nleaf_i = pl->nbox_i[lmax], nleaf_j = pl->nbox_j[lmax];
  pl->p2p_list.alloc((size_t)nleaf_i * kP2PSlots);
  p2p_lists<<<blocks((size_t)nleaf_i * kP2PSlots, 256), 256, 0, s>>>(nleaf_i, pl->key_i.get() + pl->off_i[lmax], nleaf_j,
                                                 pl->key_j.get() + pl->off_j[lmax], lmax, pl->p2p_list.get());
  FMMB_CHECK_LAUNCH();
  pl->m2l_list.alloc((size_t)pl->tot_i * kM2LSlots);
  for (int lev = 2; lev <= lmax; lev++) {
    const int nb = pl->nbox_i[lev];
    m2l_lists<<<blocks((size_t)nb * kM2LSlots, 256), 256, 0, s>>>(
        nb, pl->key_i.get() + pl->off_i[lev], pl->nbox_j[lev], pl->key_j.get() + pl->off_j[lev], lev,
        pl->d_slot_rel.get(), pl->m2l_list.get() + (size_t)pl->off_i[lev] * kM2LSlots);
    FMMB_CHECK_LAUNCH();
  }
  count_p2p_pairs<<<std::min(blocks((size_t)nleaf_i * kP2PSlots, 256), 1184), 256, 0, s>>>(nleaf_i, pl->leaf_i.get(), pl->leaf_j.get(), pl->p2p_list.get(),
                                                       cnt.get());
  FMMB_CHECK_LAUNCH();
  count_nonneg<<<std::min(blocks((size_t)pl->tot_i * kM2LSlots, 1024), 1184), 256, 0, s>>>((size_t)pl->tot_i * kM2LSlots, pl->m2l_list.get(), cnt.get() + 1);
  FMMB_CHECK_LAUNCH();
  unsigned long long h[3];
  FMMB_CUDA(cudaMemcpyAsync(h, cnt.get(), sizeof(h), cudaMemcpyDeviceToHost, s));
  FMMB_CUDA(cudaStreamSynchronize(s));
  FMMB_REQUIRE(h[2] == 0, FMMB_ERR_STATE, "tree build: inconsistent levels");
  pl->p2p_pairs = (long long)h[0];
  pl->m2l_pairs = (long long)h[1];
}

}  // namespace fmmb
