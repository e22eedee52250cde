// The source list of one near-field work item, shared by the near-field
// kernels: the leaves of the target leaf's 27 neighbour slots laid end to end
// as [own leaf | pad | others | pad], both parts padded to a multiple of 32,
// so that runs of 32 sources need no bounds check and only the own leaf's runs
// can hold a point coincident with a target (coincident points share a leaf).
#pragma once

#include <cuda_runtime.h>

#include <climits>

#include "internal.h"

namespace fmmb {

constexpr int kSelfSlot = 13;  // offset (0, 0, 0) in the 27-slot list

__device__ __forceinline__ int pad32(int n) { return (n + 31) & ~31; }

// Two points, given their coordinates' differences, are not the same one.  (Their
// squared distance does not tell: a softening is in it, and it can underflow.)
__device__ __forceinline__ bool apart(float dx, float dy, float dz) {
  return ((__float_as_int(dx) | __float_as_int(dy) | __float_as_int(dz)) & 0x7fffffff) != 0;
}

struct SrcList {
  int2 seg[32];  // (first source, count), own leaf first; slot 31: (0, sources of the others)
  int vst[32];   // virtual start of each segment, then INT_MAX

  // Called by the 32 lanes of one warp (lane l reads neighbour slot l), then a
  // block barrier: the own leaf goes first, the non-empty others after it in
  // slot order.
  __device__ __forceinline__ void build(int b, const int* __restrict__ list, const int2* __restrict__ leaf_j, int lane) {
    int2 sg = make_int2(0, 0);
    if (lane < kP2PSlots) {
      const int jl = list[(size_t)b * kP2PSlots + lane];
      if (jl >= 0) sg = leaf_j[jl];
    }
    const int self_end = pad32(__shfl_sync(0xffffffffu, sg.y, kSelfSlot));
    const bool oth = lane != kSelfSlot && sg.y > 0;
    const unsigned mask = __ballot_sync(0xffffffffu, oth);
    const int pos = 1 + __popc(mask & ((1u << lane) - 1u));
    const int cnt = oth ? sg.y : 0;
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    const int nseg = 1 + __popc(mask);
    if (lane == kSelfSlot) {
      seg[0] = sg;
      vst[0] = 0;
    }
    if (oth) {
      seg[pos] = sg;
      vst[pos] = self_end + incl - cnt;
    }
    if (lane >= nseg) vst[lane] = INT_MAX;
    const int n_other = __shfl_sync(0xffffffffu, incl, 31);
    if (lane == 0) seg[31] = make_int2(0, n_other);  // slot 31 is never a segment
  }
  __device__ __forceinline__ int self_end() const { return pad32(seg[0].y); }
  __device__ __forceinline__ int length() const { return pad32(seg[0].y) + pad32(seg[31].y); }
  // the source at virtual position v (-1: padding)
  __device__ __forceinline__ int locate(int v, int end) const {
    int sgi = 0;
#pragma unroll
    for (int st = 16; st > 0; st >>= 1)
      if (vst[sgi + st] <= v) sgi += st;
    const int2 sg = seg[sgi];
    const int off = v - vst[sgi];
    return (v < end && off < sg.y) ? sg.x + off : -1;
  }
};

}  // namespace fmmb
