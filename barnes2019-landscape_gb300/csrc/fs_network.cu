// fs_network.cu -- the drainage network of a timestep's receivers, for callers
// that read it back: levels (fastscape_RB.cpp:213-254), the Braun-Willett
// order (fastscape_BW.cpp:201-221) and the plain arrays in their ABI types.
//
// A cell's level is the length of its path to a root, and its place in the
// depth-first order is a sum along that path too: 1 + the subtrees of its
// smaller-numbered siblings at every step, and at the root the trees before
// it. So both are one pointer-jumping pass (Wyllie's list ranking) instead of
// a walk over the levels: a cell's word holds a cell further down its path
// and the sum up to there, and adding that cell's word moves it on. All words
// live in one array that is updated in place: whatever state a word is read
// in, it is a true statement about its cell, so no rounds and no barriers are
// needed, and the path still to go shrinks by half with every step of its
// cells. A walk of the levels costs a grid barrier or a launch for each: 1203
// x 1499 with 639 levels took 4.9 ms for the levels and 5.5 ms for the order.
#include <cuda_runtime.h>

#include <cstdint>

#include "fastscape_gb300.h"
#include "fs_device.h"
#include "fs_internal.h"

namespace fs {

namespace {

constexpr uint32_t kEnd = 0xFFFFFFFFu;  // the word's sum is complete
constexpr int kNetBlock = 1024;

__device__ __forceinline__ unsigned long long net_word(uint32_t next, uint32_t sum) {
  return (unsigned long long)next << 32 | sum;
}

__global__ void __launch_bounds__(256) k_net_depth(const int8_t *__restrict__ rec, int n, int W,
                                                   unsigned long long *words) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const int k = rec[i];
  words[i] = k < 0 ? net_word(kEnd, 0) : net_word((uint32_t)(i + nbr_off(k, W)), 1);
}

// Follows every cell's path. LEVELS: out[i] = its sum, and the largest one
// into rctl; else out[sum] = i. A sum grows with each step and is at most n
// unless the path runs into a cycle, which ends it with an error.
template <bool LEVELS>
__global__ void __launch_bounds__(256) k_net_follow(unsigned long long *words, int n, int32_t *out,
                                                    RealCtl *rctl, Ctl *ctl) {
  __shared__ int s_most;
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (LEVELS && threadIdx.x == 0) s_most = 0;
  if (LEVELS) __syncthreads();
  int level = 0;
  if (i < n) {
    unsigned long long w = words[i];
    uint32_t p = (uint32_t)(w >> 32), v = (uint32_t)w;
    bool moved = false, ok = v < (uint32_t)n;
    while (ok && p != kEnd) {
      const unsigned long long u = ld_relaxed_u64(words + p);
      if (moved) *reinterpret_cast<volatile unsigned long long *>(words + i) = net_word(p, v);
      p = (uint32_t)(u >> 32);
      v += (uint32_t)u;
      moved = true;
      ok = v < (uint32_t)n;
    }
    if (!ok) {
      raise_err(ctl, FS_ERR_ORDER, kPhaseOrder);
    } else {
      if (moved) *reinterpret_cast<volatile unsigned long long *>(words + i) = net_word(kEnd, v);
      out[LEVELS ? (uint32_t)i : v] = (int32_t)(LEVELS ? v : (uint32_t)i);
      level = (int)v + 1;
    }
  }
  if (LEVELS) {
    const int most = __reduce_max_sync(kFull, level);
    if ((threadIdx.x & 31) == 0) atomicMax(&s_most, most);
    __syncthreads();
    if (threadIdx.x == 0 && s_most > ld_volatile_i32(&rctl->nlevels))
      atomicMax(&rctl->nlevels, s_most);
  }
}

// Exclusive sums over the roots before a cell, of their trees' sizes (x) and
// their number (y): block totals, one block over the totals (sums[nb]: all),
// and the blocks again.
__device__ __forceinline__ int2 net_roots(const int8_t *rec, const uint32_t *count, int i, int n,
                                          int2 &total) {
  const bool root = i < n && rec[i] < 0;
  int2 before;
  before.x = block_excl_scan(root ? (int)count[i] : 0, total.x, threadIdx.x, kNetBlock);
  __syncthreads();
  before.y = block_excl_scan(root ? 1 : 0, total.y, threadIdx.x, kNetBlock);
  return before;
}

__global__ void __launch_bounds__(kNetBlock) k_net_root_sums(const int8_t *__restrict__ rec,
                                                             const uint32_t *__restrict__ count,
                                                             int n, int2 *sums) {
  int2 total;
  net_roots(rec, count, blockIdx.x * kNetBlock + threadIdx.x, n, total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kNetBlock) k_net_scan(int2 *sums, int nb) {
  const int per = (nb + kNetBlock - 1) / kNetBlock;
  const int b0 = threadIdx.x * per, b1 = min(b0 + per, nb);
  int2 s = make_int2(0, 0), total, run;
  for (int b = b0; b < b1; b++) {
    s.x += sums[b].x;
    s.y += sums[b].y;
  }
  run.x = block_excl_scan(s.x, total.x, threadIdx.x, kNetBlock);
  __syncthreads();
  run.y = block_excl_scan(s.y, total.y, threadIdx.x, kNetBlock);
  for (int b = b0; b < b1; b++) {
    const int2 x = sums[b];
    sums[b] = run;
    run.x += x.x;
    run.y += x.y;
  }
  if (threadIdx.x == 0) sums[nb] = total;
}

// The depth-first order's words, and where each tree starts. A receiver's
// donors come in ascending cell order (fastscape_BW.cpp:188-198); count is
// the drainage count, which is the size of a cell's subtree.
__global__ void __launch_bounds__(kNetBlock) k_net_order(const int8_t *__restrict__ rec,
                                                         const uint32_t *__restrict__ count, int n,
                                                         int W, const int2 *__restrict__ sums,
                                                         unsigned long long *words,
                                                         int32_t *starts) {
  const int i = blockIdx.x * kNetBlock + threadIdx.x;
  int2 total;
  const int2 before = net_roots(rec, count, i, n, total);
  if (i >= n) return;
  const int k = rec[i];
  if (k < 0) {
    const int at = sums[blockIdx.x].x + before.x;
    starts[sums[blockIdx.x].y + before.y] = at;
    words[i] = net_word(kEnd, (uint32_t)at);
    return;
  }
  const int p = i + nbr_off(k, W), x = p % W;
  uint32_t sum = 1;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    // the cells before p + 1 around p: its N row, west to east, and W
    const int dir = j < 3 ? 1 + j : 0;
    const int q = p + nbr_off(dir, W);
    const bool there = q >= 0 && !(x == 0 && (dir == 0 || dir == 1)) && !(x == W - 1 && dir == 3);
    if (there && q < i && rec[q] == dir + 4) sum += count[q];
  }
#pragma unroll
  for (int dir = 4; dir < 7; dir++) {
    // and those before its SE neighbour: E, and S's row (7 SW, 6 S)
    const int d = dir == 4 ? 4 : dir == 5 ? 7 : 6;
    const int q = p + nbr_off(d, W);
    const bool there = q < n && !(x == W - 1 && d == 4) && !(x == 0 && d == 7);
    if (there && q < i && rec[q] == d - 4) sum += count[q];
  }
  words[i] = net_word((uint32_t)p, sum);
}

// The ABI's types: receivers (as FS_NO_FLOW or a direction), their cells (the
// cell itself without one) and drained areas.
__global__ void __launch_bounds__(256) k_net_receivers(const int8_t *__restrict__ rec, int n,
                                                       int32_t *out) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) out[i] = rec[i] < 0 ? FS_NO_FLOW : rec[i];
}

__global__ void __launch_bounds__(256) k_net_receiver_index(const int8_t *__restrict__ rec, int n,
                                                            int W, long long *out) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) out[i] = rec[i] < 0 ? i : i + nbr_off(rec[i], W);
}

__global__ void __launch_bounds__(256) k_net_area(const uint32_t *__restrict__ count, int n,
                                                  double cell_area, double *out) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) out[i] = __dmul_rn((double)count[i], cell_area);
}

int blocks(int n, int per) { return (int)(((long long)n + per - 1) / per); }

}  // namespace

cudaError_t launch_net_levels(const NetArgs &a, RealCtl *rctl, Ctl *ctl, int32_t *out,
                              cudaStream_t s) {
  k_net_depth<<<blocks(a.n, 256), 256, 0, s>>>(a.rec, a.n, a.W, a.words);
  k_net_follow<true><<<blocks(a.n, 256), 256, 0, s>>>(a.words, a.n, out, rctl, ctl);
  return cudaGetLastError();
}

cudaError_t launch_net_trees(const NetArgs &a, int2 *sums, int32_t *starts, cudaStream_t s) {
  const int nb = blocks(a.n, kNetBlock);
  k_net_root_sums<<<nb, kNetBlock, 0, s>>>(a.rec, a.count, a.n, sums);
  k_net_scan<<<1, kNetBlock, 0, s>>>(sums, nb);
  k_net_order<<<nb, kNetBlock, 0, s>>>(a.rec, a.count, a.n, a.W, sums, a.words, starts);
  return cudaGetLastError();
}

cudaError_t launch_net_order(const NetArgs &a, Ctl *ctl, int32_t *out, cudaStream_t s) {
  k_net_follow<false><<<blocks(a.n, 256), 256, 0, s>>>(a.words, a.n, out, nullptr, ctl);
  return cudaGetLastError();
}

int net_sums(int n) { return blocks(n, kNetBlock); }

cudaError_t launch_net_receivers(const NetArgs &a, int32_t *out, cudaStream_t s) {
  k_net_receivers<<<blocks(a.n, 256), 256, 0, s>>>(a.rec, a.n, out);
  return cudaGetLastError();
}

cudaError_t launch_net_receiver_index(const NetArgs &a, long long *out, cudaStream_t s) {
  k_net_receiver_index<<<blocks(a.n, 256), 256, 0, s>>>(a.rec, a.n, a.W, out);
  return cudaGetLastError();
}

cudaError_t launch_net_area(const NetArgs &a, double cell_area, double *out, cudaStream_t s) {
  k_net_area<<<blocks(a.n, 256), 256, 0, s>>>(a.count, a.n, cell_area, out);
  return cudaGetLastError();
}

}  // namespace fs
