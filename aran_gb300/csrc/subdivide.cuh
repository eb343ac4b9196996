// subdivide.cuh -- the internal nodes of an octree or quadtree from its sorted
// keys (tree.cu, solver2d.cu).
#pragma once
#include "internal.cuh"

namespace aran {
namespace {

// ---------------------------------------------------------------------------
// Subdivision of all levels at once.  A node of depth d holds the particles
// that share the first d digits of their keys (within a system).  One starts at
// sorted place i if d exceeds the digits that places i - 1 and i share, and has
// more than maxbox points if places i and i + maxbox share d: the internal nodes
// that start at i are those of the depths lo .. hi.  Counted per depth and block
// of places and scanned depth by depth, their numbers are their ranks in level
// order, the children of the node of rank r in its level lie at eight (2D: four) times
// r in the next, and one readback (the counts) is all that the host waits for;
// level by level each took one, with a flag pass, a scan and a binary search
// of its own: 40 us a level.  Bound by latency: 10k uniform particles (4 levels)
// 0.056 ms, 0.165 before; 4M Plummer particles (11 levels) 0.115 ms, 0.524.
// ---------------------------------------------------------------------------
constexpr int kPlaceBlock = 256, kPlaceItems = 4, kPlaces = kPlaceBlock * kPlaceItems;
constexpr int kPlaceSlots = kPlaces / 32;   // warp-wide runs of places in a block
static_assert(kPlaceSlots == 32, "a warp scans a block's slots");

// counts[d][block]: internal nodes of depth d that start in the block's places
template <typename Keys>
__global__ void __launch_bounds__(kPlaceBlock) k_count_internal(Keys keys, int *__restrict__ counts) {
  __shared__ int cnt[kKeyBits][kPlaceSlots + 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int c = 0; c < kPlaceItems; ++c) {
    int lo, hi, v = 0;
    keys.internal_depths((int64_t)blockIdx.x * kPlaces + c * kPlaceBlock + threadIdx.x, lo, hi);
    const int d0 = __reduce_min_sync(0xffffffffu, lo), d1 = __reduce_max_sync(0xffffffffu, hi);
    for (int d = d0; d <= d1; ++d) {
      const unsigned m = __ballot_sync(0xffffffffu, lo <= d && d <= hi);
      if (lane == d) v = __popc(m);
    }
    if (lane < kKeyBits) cnt[lane][c * (kPlaceBlock / 32) + w] = v;
  }
  __syncthreads();
  for (int d = w; d < kKeyBits; d += kPlaceBlock / 32) {
    const int t = __reduce_add_sync(0xffffffffu, cnt[d][lane]);
    if (lane == 0) counts[(int64_t)d * gridDim.x + blockIdx.x] = t;
  }
}

// place and parent's rank of every internal node, by rank in level order
template <typename Keys>
__global__ void __launch_bounds__(kPlaceBlock)
    k_list_internal(Keys keys, const int *__restrict__ first, int *__restrict__ start,
                    int *__restrict__ prank) {
  __shared__ int pre[kKeyBits][kPlaceSlots + 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int lo[kPlaceItems], hi[kPlaceItems];
#pragma unroll
  for (int c = 0; c < kPlaceItems; ++c) {
    int v = 0;
    keys.internal_depths((int64_t)blockIdx.x * kPlaces + c * kPlaceBlock + threadIdx.x, lo[c],
                         hi[c]);
    const int d0 = __reduce_min_sync(0xffffffffu, lo[c]), d1 = __reduce_max_sync(0xffffffffu, hi[c]);
    for (int d = d0; d <= d1; ++d) {
      const unsigned m = __ballot_sync(0xffffffffu, lo[c] <= d && d <= hi[c]);
      if (lane == d) v = __popc(m);
    }
    if (lane < kKeyBits) pre[lane][c * (kPlaceBlock / 32) + w] = v;
  }
  __syncthreads();
  // ranks before each run of places
  for (int d = w; d < kKeyBits; d += kPlaceBlock / 32) {
    const int mine = pre[d][lane];
    int v = mine;
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    pre[d][lane] = first[(int64_t)d * gridDim.x + blockIdx.x] + v - mine;
  }
  __syncthreads();
  const unsigned before = (1u << lane) - 1;
#pragma unroll
  for (int c = 0; c < kPlaceItems; ++c) {
    const int slot = c * (kPlaceBlock / 32) + w;
    const int64_t i = (int64_t)blockIdx.x * kPlaces + c * kPlaceBlock + threadIdx.x;
    const int d0 = __reduce_min_sync(0xffffffffu, lo[c]), d1 = __reduce_max_sync(0xffffffffu, hi[c]);
    unsigned up = 0;                     // the depth above's starts in this run
    for (int d = d0; d <= d1; ++d) {
      const unsigned m = __ballot_sync(0xffffffffu, lo[c] <= d && d <= hi[c]);
      if (lo[c] <= d && d <= hi[c]) {
        const int rk = pre[d][slot] + __popc(m & before);
        start[rk] = (int)i;
        if (d > 0) prank[rk] = pre[d - 1][slot] + __popc(up & (before | 1u << lane)) - 1;
      }
      up = m;
    }
  }
}

// first rank and first node of each depth (by value to the kernel)
struct LevelStarts {
  int rank[kKeyBits + 1], node[kKeyBits + 2];
};

// The host side: counts of all depths scanned into first[d][block] (kKeyBits
// rows of nb, then the total; `work` holds as many ints), first ranks copied to hb[0 ..
// kKeyBits] (the caller waits).  Returns the blocks nb.
inline int place_blocks(int64_t n) { return (int)((n + kPlaces - 1) / kPlaces); }

template <typename Keys, typename Scan>
void count_internal(const Keys &keys, int nb, int *work, int *first, int *hb, Scan &&scan,
                    cudaStream_t st) {
  const int nc = kKeyBits * nb;
  k_count_internal<<<nb, kPlaceBlock, 0, st>>>(keys, work);
  ACHECK(cudaGetLastError());
  ACHECK(cudaMemsetAsync(work + nc, 0, sizeof(int), st));
  scan(work, first, nc + 1);
  ACHECK(cudaMemcpy2DAsync(hb, sizeof(int), first, nb * sizeof(int), sizeof(int), kKeyBits + 1,
                           cudaMemcpyDeviceToHost, st));
}

// levels from the first ranks hb: nodes per level (fan children each), starts
inline LevelStarts level_starts(const int *hb, int nsys, int fan, std::vector<int> &level_off,
                                std::vector<int> *level_internal) {
  LevelStarts ls = {};
  level_off.assign(1, 0);
  int off = 0, cnt = nsys, d = 0;
  for (; cnt > 0; ++d) {
    ls.node[d] = off;
    off += cnt;
    level_off.push_back(off);
    const int ninternal = d < kKeyBits ? hb[d + 1] - hb[d] : 0;
    if (level_internal) level_internal->push_back(ninternal);
    cnt = fan * ninternal;
  }
  for (int k = 0; k <= kKeyBits; ++k) ls.rank[k] = hb[k];
  for (int k = d; k < kKeyBits + 2; ++k) ls.node[k] = off;
  return ls;
}

}  // namespace
}  // namespace aran
