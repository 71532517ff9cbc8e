// fs_tile.cu -- the tile walk: flow accumulation (fastscape_RB.cpp:262-279),
// uplift (:285-296) and implicit erosion (:306-328) of a timestep from its
// receivers, in 64 x 32 tiles whose working set stays in shared memory.
//
// The reference orders all cells by their depth in the drainage forest and
// sweeps the levels. A grid-wide sweep costs a grid barrier and a chain of
// dependent memory accesses per level (3-4 us in each of three kernels: 2.7
// ms per timestep of an eroded 512^2 grid, 265 levels deep), and it gathers
// every operand from the level order (23 warp instructions a cell at
// 10000^2). Only what crosses a tile's edge needs more than one SM, and that
// is little: on the 10000^2 workload's ground 2.6% of the cells drain into
// another tile and 4.0% lie upstream of such a cell; on deeply eroded ground
// a path of 280 cells crosses at most 20 edges. So:
//   1. k_tile_drain   per tile: the cells each cell drains inside the tile,
//                     and where water entering the tile leaves it again;
//   2. k_tile_links   drainage handed from tile to tile along those links;
//   3. where every tile of the launch is on the GPU at once,
//      k_tile_resident  per tile: adds the water from outside, then uplifts
//                       and erodes, the trees that hang on other tiles as
//                       their receivers become final;
//   4. otherwise
//      k_tile_rooted    the same for the trees rooted in the tile,
//      k_tile_pull      (n = 1) the cells of short paths into other tiles, each
//                       by itself (k_tile_mark tells the queue),
//      k_tile_front     (n != 1, or many cells left) cells in rounds of the
//                       whole GPU,
//      k_tile_queue     what is left, from a queue of tiles.
// Counts are sums of integers, exact in any order, and a cell is eroded by
// the same operations from the same operands as in the reference's order, so
// every result is the same bit for bit.
#include <cuda_runtime.h>

#include <cstdint>

#include "fastscape_gb300.h"
#include "fs_bits.h"
#include "fs_device.h"
#include "fs_internal.h"

namespace fs {

namespace {

constexpr int kDrainThreads = 256;
constexpr int kWalkThreads = 128;  // a warp that finds the levels, 3 that erode
// Of k_tile_resident's blocks: 6, 4 and 2 share an SM (80 registers a thread).
constexpr int kResidentThreads[kResidentWidths] = {128, 192, 384};
constexpr int kCore = 96;          // threads that erode every level
// Levels found ahead of the erosion, at most. What a neighbour makes ready is
// eroded behind them: 501^2 with n = 2 takes 1130 us at 6, 1070 at 4, 1036 at
// 3 and 1041 at 2, where eroded 512^2 begins to wait for the finder (617 us
// against 607).
constexpr int kLead = 3;
constexpr int kRing = 8;           // level ends and rows kept
constexpr int kStageFrom = 256;    // unfinished cells worth staging a tile for
constexpr int kPullMost = 256;     // unfinished cells k_tile_pull takes from a tile, at most
constexpr int kPullDepth = 16;     // and how far up it follows their receivers
constexpr int kPullThreads = 96;
constexpr int kRootedThreads = 192;
constexpr int kFrontThreads = 384;
// n = 1: cells of trees that leave their tile from which k_tile_front takes
// them. 256 realizations of eroded 512^2, 60e6 such cells, take 11.9 ms a
// timestep with the queue alone and 7.6 so; eroded 2000^2, 3e6, 1.36 and 1.40.
constexpr int kFrontCells = 1 << 23;
// Rounds too narrow for the GPU's threads end when more than so many would
// follow: 10000^2 with n = 2, 65 levels, takes 7.26 ms a timestep at 4 and 8 and
// 7.00 at 16; ended by width alone, 7.21 below 2048 cells and 7.24 below 131072,
// with n = 1.5 and 12 levels 36.5 below 131072 (35.7 at 4 to 16).
constexpr int kFrontRounds = 16;
// n != 1: a tile's levels narrower than this are left to k_tile_front, which
// has full warps for them. n = 2: 7.00 -> 6.85 ms at 48 (96: 6.80, but 13.5
// instead of 12.7 at 515 levels; 192: 7.07). Other n, whose cells take five times
// as long: 35.7 -> 34.5 at 192 (48: 34.8, 400: 34.6, every level: 35.1), and
// every level where the tiles come in few waves (672 x 4422, 1518 tiles, 1.44 ->
// 1.39; 1500^2 1.15 -> 1.09; 3000^2, 4418 tiles, 3.41 -> 3.52).
constexpr int kRootedFewTwo = 48, kRootedFewGeneral = 192, kRootedWaves = 4096;
static_assert(kWalkW == 64 && kWalkH == 32, "a cell's tile: x >> 6, y >> 5");
constexpr uint32_t kNoSink = 0xFFFFu;
constexpr int kFinished = 1 << 30;
constexpr int kTileQueued = 1, kTileAgain = 2;
enum Mode { kResident = 1, kQueued = 2 };

// Offset of direction k inside a tile: a byte of two packed words (+65).
__device__ __forceinline__ int tile_off(int k) {
  return (int)(__byte_perm(0x02010040u, 0x80818242u, k) & 0xFFu) - 65;
}

__device__ __forceinline__ int slot_cell(int s) {
  if (s < 64) return s;
  if (s < 128) return (kWalkH - 1) * 64 + s - 64;
  return s < 160 ? (s - 128) * 64 : (s - 160) * 64 + 63;
}

// Perimeter slot of a cell on the tile's edge.
__device__ __forceinline__ int cell_slot(int c) {
  const int x = c & 63, y = c >> 6;
  if (y == 0) return x;
  if (y == kWalkH - 1) return 64 + x;
  return x == 0 ? 128 + y : 160 + y;
}

// The corners lie in rows and columns; the rows' slots name them.
__device__ __forceinline__ bool slot_valid(int s) {
  return s < 128 || ((s & 31) != 0 && (s & 31) != kWalkH - 1);
}

__device__ __forceinline__ int tile_of(const StepArgs &a, int i) {
  return a.tb.list ? a.tb.list[i] : i;
}

__device__ __forceinline__ int dir_dx(int k) { return ((0x1A90 >> (2 * k)) & 3) - 1; }
__device__ __forceinline__ int dir_dy(int k) { return ((0xA901 >> (2 * k)) & 3) - 1; }

// Target of an exit at cell c in direction k: neighbour tile (dy+1)*3 + dx+1
// and the slot the water enters it at.
__device__ __forceinline__ uint32_t exit_target(int c, int k) {
  const int nx = (c & 63) + dir_dx(k), ny = (c >> 6) + dir_dy(k);
  const int tx = nx < 0 ? -1 : nx > 63 ? 1 : 0, ty = ny < 0 ? -1 : ny >= kWalkH ? 1 : 0;
  const int slot = cell_slot(((ny & (kWalkH - 1)) << 6) | (nx & 63));
  return (uint32_t)(((ty + 1) * 3 + tx + 1) << 8 | slot);
}

// ---------------------------------------------------------------------------
// 1. Drainage inside a tile.
//
// Each cell's shared word holds the cells it drains so far (low half, 1 at
// first) and the receivers' donors still to come (high half). The cells
// without a donor in the tile (72% of young ground) add their count to their
// receiver's word and take one off its donors, in one shared-memory atomic;
// a cell whose last donor has come goes on a list, and the list's cells do the
// same, round after round, with full warps (the last short rounds in one
// warp). Every cell is handled once, and no order of the cells is needed.
// Then the edge: a cell that water of another tile enters leads to one sink
// (the exit it leaves by, or the cell above the root it ends in), and an exit
// knows how many edges lead into its tree from outside.
//
// A thread has eight cells of a row: their codes come as three aligned words,
// and the bit planes' bytes from one multiplication each. The shared words
// are padded (one in nine unused), so that eight consecutive words a thread
// meet no bank conflict.
// ---------------------------------------------------------------------------
constexpr int kPadded = kWalkCells + kWalkCells / 8;

__device__ __forceinline__ int padded(int c) { return c + (c >> 3); }

__global__ void __launch_bounds__(kDrainThreads) k_tile_drain(StepArgs a) {
  if (stopped(a.ctl)) return;
  if (threadIdx.x == 0) {
    a.tb.queue[blockIdx.x] = 0;  // a ring of the launch's own n places, whatever tiles it lists
    if (blockIdx.x == 0) {       // for this timestep's walk and the next's filter
      a.ctl->amb = 0;
      a.ctl->left = a.ctl->progress = 0;
      a.ctl->qtail = a.ctl->qhead = 0;
      a.ctl->bar = a.ctl->front[0] = a.ctl->front[1] = 0;
    }
  }
  __shared__ __align__(16) uint32_t s_w[kPadded];
  __shared__ __align__(16) uint8_t s_code[kWalkCells];
  __shared__ __align__(16) uint8_t s_plane[4 * 256];
  __shared__ uint16_t s_list[kWalkCells];
  __shared__ uint32_t s_pend[kSlots];
  __shared__ int8_t s_halo[2 * (kWalkW + 2) + 2 * kWalkH];  // above, below, left, right
  __shared__ int s_nstart;
  __shared__ int s_cnt[3];  // cells a round lists (rotating)
  static_assert(kWalkCells == 8 * kDrainThreads, "eight cells a thread");
  constexpr int kBelow = kWalkW + 2, kLeft = 2 * kBelow, kRight = kLeft + kWalkH;
  const int t = tile_of(a, blockIdx.x);
  const Tile tl = a.tb.tiles[t];
  const RealDesc &d = a.tb.desc[tl.r];
  const int W = d.W, H = d.H;
  const int8_t *rec = a.rec + d.off;
  const int tid = threadIdx.x, lane = tid & 31;
  const int y = tid >> 3, xb = tid & 7;
  // The thread's eight codes, as the bytes of lo and hi. The aligned words
  // around them lie within the padding of rec.
  const int inside = tl.y0 + y < H ? min(max(W - tl.x0 - 8 * xb, 0), 8) : 0;
  uint32_t lo = 0, hi = 0;
  if (inside > 0) {
    const uintptr_t p = reinterpret_cast<uintptr_t>(rec + (size_t)(tl.y0 + y) * W + tl.x0 + 8 * xb);
    const uint32_t *w = reinterpret_cast<const uint32_t *>(p & ~(uintptr_t)3);
    const int sh = (int)(p & 3) * 8;
    const uint32_t w0 = __ldg(w), w1 = __ldg(w + 1), w2 = __ldg(w + 2);
    lo = __funnelshift_r(w0, w1, sh);
    hi = __funnelshift_r(w1, w2, sh);
  }
  int8_t halo = (int8_t)FS_NO_FLOW;
  if (tid < kRight + kWalkH) {
    int hx, hy;
    if (tid < kLeft) {
      hx = tl.x0 - 1 + (tid < kBelow ? tid : tid - kBelow);
      hy = tid < kBelow ? tl.y0 - 1 : tl.y0 + kWalkH;
    } else {
      hx = tid < kRight ? tl.x0 - 1 : tl.x0 + kWalkW;
      hy = tl.y0 + (tid < kRight ? tid - kLeft : tid - kRight);
    }
    if (hx >= 0 && hy >= 0 && hx < W && hy < H) halo = __ldg(rec + (size_t)hy * W + hx);
  }
  for (int i = tid; i < kPadded / 4; i += kDrainThreads)
    reinterpret_cast<uint4 *>(s_w)[i] = make_uint4(1u, 1u, 1u, 1u);
  if (tid < kSlots) s_pend[tid] = 0;
  if (tid < 3) s_cnt[tid] = 0;
  if (tid == 3) s_nstart = 0;
  if (tid < kRight + kWalkH) s_halo[tid] = halo;
  {
    // no receiver (negative): kCodeRoot; past the grid: kCodeOutside
    const uint32_t nl = (lo & 0x80808080u) >> 7, nh = (hi & 0x80808080u) >> 7;
    uint32_t fl = nl ^ 0x01010101u, fh = nh ^ 0x01010101u;  // has a receiver
    lo = (lo & ~(nl * 255u)) | nl * kCodeRoot;
    hi = (hi & ~(nh * 255u)) | nh * kCodeRoot;
    if (inside < 8) {
      const uint32_t ol = inside >= 4 ? 0u : 0xFFFFFFFFu << (8 * inside);
      const uint32_t oh = inside <= 4 ? 0xFFFFFFFFu : 0xFFFFFFFFu << (8 * inside - 32);
      lo = (lo & ~ol) | (ol & (0x01010101u * kCodeOutside));
      hi = (hi & ~oh) | (oh & (0x01010101u * kCodeOutside));
      fl &= ~ol;
      fh &= ~oh;
    }
    // bit p of the eight bytes as one byte: the product moves the bits at 0,
    // 8, 16, 24 to 24..27 and those at 4, 12, 20, 28 to 28..31
    auto pack = [](uint32_t l, uint32_t h) { return (uint8_t)((l | h << 4) * 0x01020408u >> 24); };
#pragma unroll
    for (int p = 0; p < 3; p++) s_plane[p * 256 + tid] = pack(lo >> p & fl, hi >> p & fh);
    s_plane[3 * 256 + tid] = pack(fl, fh);
    // exits: directions that leave the tile
    auto mark = [](uint32_t &w, int b, unsigned out) {
      const uint32_t c = w >> (8 * b) & 0xFFu;
      if (c < 8 && (out >> c & 1u)) w |= (uint32_t)kCodeExit << (8 * b);
    };
    if (xb == 0) mark(lo, 0, 0x83u);
    if (xb == 7) mark(hi, 3, 0x38u);
    if (y == 0 || y == kWalkH - 1) {
      const unsigned out = y == 0 ? 0x0Eu : 0xE0u;
#pragma unroll
      for (int b = 0; b < 4; b++) {
        mark(lo, b, out);
        mark(hi, b, out);
      }
    }
    reinterpret_cast<uint2 *>(s_code)[tid] = make_uint2(lo, hi);
  }
  __syncthreads();
  int r[8];            // receivers' words
  unsigned in = 0;     // cells with a receiver in the tile
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const int k = (int)((j < 4 ? lo : hi) >> (8 * (j & 3)) & 0xFFu);
    r[j] = 0;
    if (k < 8) {
      r[j] = 8 * tid + j + tile_off(k);
      atomicAdd(&s_w[padded(r[j])], 1u << 16);
      in |= 1u << j;
    }
  }
  __syncthreads();
  unsigned leaves = 0;
#pragma unroll
  for (int j = 0; j < 8; j++)
    if (s_w[9 * tid + j] >> 16 == 0) leaves |= 1u << j;
  leaves &= in;
  __syncthreads();  // every leaf is known before the first count moves
  unsigned last = 0;
#pragma unroll
  for (int j = 0; j < 8; j++)
    if (leaves >> j & 1u)
      last |= (atomicAdd(&s_w[padded(r[j])], 1u - (1u << 16)) >> 16 == 1 ? 1u : 0u) << j;
  {
    const int n = __popc(last);
    int incl = n;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const int v = __shfl_up_sync(kFull, incl, s);
      if (lane >= s) incl += v;
    }
    int at = 0;
    if (lane == 31 && incl) at = atomicAdd(&s_cnt[0], incl);
    at = __shfl_sync(kFull, at, 31) + incl - n;
#pragma unroll
    for (int j = 0; j < 8; j++)
      if (last >> j & 1u) s_list[at++] = (uint16_t)r[j];
  }
  // a listed cell passes its count on; the receiver, if that was its last
  // donor, else -1
  auto pass = [&](int i) -> int {
    const int c = s_list[i], k = s_code[c];
    if (k >= 8) return -1;  // a root, or an exit: the rest of the path is elsewhere
    const int to = c + tile_off(k);
    const uint32_t v = s_w[padded(c)] & 0xFFFFu;
    return atomicAdd(&s_w[padded(to)], v - (1u << 16)) >> 16 == 1 ? to : -1;
  };
  __syncthreads();
  int b = 0, e = s_cnt[0];
  for (int round = 1; e - b > 64; ++round) {
    int *cnt = &s_cnt[round % 3];
    if (tid == 0) s_cnt[(round + 1) % 3] = 0;
    for (int i = b + (tid & ~31); i < e; i += kDrainThreads) {
      const int to = i + lane < e ? pass(i + lane) : -1;
      const unsigned m = __ballot_sync(kFull, to >= 0);
      int at = 0;
      if (lane == 0 && m) at = atomicAdd(cnt, __popc(m));
      at = __shfl_sync(kFull, at, 0) + e + __popc(m & ((1u << lane) - 1u));
      if (to >= 0) s_list[at] = (uint16_t)to;
    }
    __syncthreads();
    b = e;
    e += *cnt;
  }
  if (tid < 32) {
    while (b < e) {
      int at = e;
      for (int i = b; i < e; i += 32) {
        const int to = i + lane < e ? pass(i + lane) : -1;
        const unsigned m = __ballot_sync(kFull, to >= 0);
        if (to >= 0) s_list[at + __popc(m & ((1u << lane) - 1u))] = (uint16_t)to;
        at += __popc(m);
      }
      __syncwarp();
      b = e;
      e = at;
    }
  }
  __syncthreads();
  {
    uint32_t w[8];
#pragma unroll
    for (int j = 0; j < 8; j++) w[j] = s_w[9 * tid + j] & 0xFFFFu;
    reinterpret_cast<uint4 *>(a.tb.local + (size_t)t * kWalkCells)[tid] =
        make_uint4(w[0] | w[1] << 16, w[2] | w[3] << 16, w[4] | w[5] << 16, w[6] | w[7] << 16);
    if (tid < kWalkCells / 16)
      reinterpret_cast<uint4 *>(a.tb.code + (size_t)t * kWalkCells)[tid] =
          reinterpret_cast<const uint4 *>(s_code)[tid];
    else if (tid < kWalkCells / 16 + 64)
      reinterpret_cast<uint4 *>(a.tb.planes + (size_t)t * 256)[tid - kWalkCells / 16] =
          reinterpret_cast<const uint4 *>(s_plane)[tid - kWalkCells / 16];
    else if (tid < kWalkCells / 16 + 64 + kWalkH)
      a.tb.done[(size_t)t * kWalkH + tid - kWalkCells / 16 - 64] = 0;
  }
  // The edge: thread s has the cell of slot s.
  const bool edge = tid < kSlots && slot_valid(tid);
  const int c0 = edge ? slot_cell(tid) : 0;
  const int code0 = edge ? s_code[c0] : kCodeOutside;
  uint32_t ext = 0;  // donors in other tiles: three beyond the slot's side ...
  if (edge && code0 != kCodeOutside) {
    const int at = tid < 64 ? tid : tid < 128 ? kBelow + tid - 64
                   : tid < 160 ? kLeft + tid - 129 : kRight + tid - 161;
    // ... whose directions are SE S SW, NE N NW, SE E NE or SW W NW
    const int want = tid < 64 ? 0x765 : tid < 128 ? 0x123 : tid < 160 ? 0x345 : 0x107;
#pragma unroll
    for (int q = 0; q < 3; q++) ext += s_halo[at + q] == (want >> (4 * q) & 7) ? 1u : 0u;
    const int sx = tid & 63;
    if (tid < 128 && (sx == 0 || sx == 63)) {  // a corner: two more beside it
      const int side = sx == 0 ? kLeft : kRight, row = tid < 64 ? 0 : kWalkH - 1;
      const int in_row = sx == 0 ? 4 : 0;                                // E or W
      const int slant = sx == 0 ? (row ? 5 : 3) : (row ? 7 : 1);         // SE NE, SW NW
      ext += s_halo[side + row] == in_row ? 1u : 0u;
      ext += s_halo[side + (row ? row - 1 : 1)] == slant ? 1u : 0u;
    }
  }
  __syncthreads();  // the counts are written out: high halves are free
  uint32_t link = kNoSink;
  int head = -1;
  if (ext) {
    int c = c0, above = -1, k = code0;
    for (int n = 0; k < 8 && n < kWalkCells; n++) {
      above = c;
      c += tile_off(k);
      k = s_code[c];
    }
    if (k >= kCodeExit) {
      link = (uint32_t)cell_slot(c) | exit_target(c, k & 7) << 16;
      atomicAdd(&s_pend[link & 0xFFFFu], ext);
    } else if (above >= 0) {  // the slots that share a head agree on the largest
      head = padded(above);
      atomicMax(&s_w[head], (uint32_t)(tid + 1) << 16 | (s_w[head] & 0xFFFFu));
    }
  }
  __syncthreads();
  unsigned long long *sink = a.tb.sink + (size_t)t * (2 * kSlots);
  if (head >= 0) {
    const uint32_t w = s_w[head];
    const int rep = (int)(w >> 16) - 1;
    link = (uint32_t)(kSlots + rep);
    if (rep == tid) sink[kSlots + rep] = (unsigned long long)(w & 0xFFFFu) << 16;
  }
  if (ext) a.tb.link[(size_t)t * kSlots + tid] = link;
  if (tid < kSlots) a.tb.inflow[(size_t)t * kSlots + tid] = 0;
  bool starts = false;
  uint32_t start = 0;
  if (code0 >= kCodeExit) {
    const uint32_t cnt = s_w[padded(c0)] & 0xFFFFu;
    sink[tid] = (unsigned long long)cnt << 16 | s_pend[tid];
    starts = s_pend[tid] == 0;
    start = exit_target(c0, code0 & 7) << 16 | cnt;
  }
  const unsigned sb = __ballot_sync(kFull, starts);
  int at = 0;
  if (lane == 0 && sb) at = atomicAdd(&s_nstart, __popc(sb));
  at = __shfl_sync(kFull, at, 0) + __popc(sb & ((1u << lane) - 1u));
  if (starts) a.tb.start[(size_t)t * kSlots + at] = start;
  __syncthreads();
  if (tid == 0) {
    a.tb.nstart[t] = s_nstart;
    a.tb.state[t] = 0;
  }
}

// ---------------------------------------------------------------------------
// 2. Drainage between tiles: an exit whose tree nothing (more) flows into
// hands its count to the entry of the next tile and to that entry's sink; the
// last one to reach a sink carries its sum on. One warp per tile; a hop is a
// load and an atomic in L2. A count beyond its realization's erosion table
// (an exit's, or the largest below a root, whose own count needs no record)
// stops the timestep before any elevation changes.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_tile_links(StepArgs a) {
  if (stopped(a.ctl)) return;
  const int lane = threadIdx.x & 31;
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= a.tb.n) return;
  const int t0 = tile_of(a, w);
  const Tile tl = a.tb.tiles[t0];
  const int cap = a.tb.desc[tl.r].tab_cap;
  const int n = a.tb.nstart[t0];
  int most = 0;
  for (int i = lane; i < n; i += 32) {
    const uint32_t st = a.tb.start[(size_t)t0 * kSlots + i];
    int t = t0;
    uint32_t v = st & 0xFFFFu, tgt = st >> 16;
    for (;;) {
      most = max(most, (int)v);
      const int nb = (int)(tgt >> 8);
      t += (nb / 3 - 1) * tl.ntx + nb % 3 - 1;
      const size_t at = (size_t)t * kSlots + (tgt & 0xFFu);
      const uint32_t l = __ldg(a.tb.link + at);
      atomicAdd(a.tb.inflow + at, v);
      const uint32_t sid = l & 0xFFFFu;
      if (sid == kNoSink) break;
      unsigned long long *sk = a.tb.sink + (size_t)t * (2 * kSlots) + sid;
      if (sid >= (uint32_t)kSlots) {
        const unsigned long long old = atomicAdd(sk, (unsigned long long)v << 16);
        most = max(most, (int)(uint32_t)((old >> 16) + v));
        break;
      }
      const unsigned long long old = atomicAdd(sk, ((unsigned long long)v << 16) - 1ull);
      if ((old & 0xFFFFull) != 1) break;
      v += (uint32_t)(old >> 16);
      tgt = l >> 16;
    }
  }
  if (a.do_erode && most >= cap) {
    if (atomicMax(&a.ctl->abort_k, most) < most) a.ctl->abort_r = tl.r;
  }
}

// ---------------------------------------------------------------------------
// 3. Erosion, level by level inside a tile. Warp 0 finds the levels: it holds
// the tile's cells as bit rows, one row per lane, and per direction the cells
// that drain that way, so the donors of a set of cells are eight shifts and
// masks; it writes their cell numbers to a list, rows in order. It runs up to
// kLead levels ahead of the other warps, which erode the cells of a level and
// meet at a barrier of their own. On young ground one level holds half of a
// tile: where the SMs have room for wider blocks, more warps sleep at another
// barrier and help with the levels wider than two rounds of the first three
// (100^2: 70 -> 57 us a timestep, 1000^2: 96 -> 87; with the steps after it 54
// and 82), which deep ground's narrow levels do not wait for. What takes time is the chain of one cell's
// arithmetic after its receiver's elevation is known (64 clocks for an FP64
// operation, four to eight of them, and the quotient's integer steps), once a
// level: everything else of a cell -- its elevation, count, table record, an
// exit's receiver -- is loaded before the barrier.
//
// kResident: all tiles of the launch are on the GPU at once; warp 0 also looks
// for exits whose receiver in a neighbouring tile has become final (its rows
// of final cells are in global memory) and adds them to the next level, and
// publishes this tile's. kQueued: exits that are ready when the tile's turn
// comes, or become so meanwhile. k_tile_rooted goes by the same steps in lock
// step, warp 0 two levels ahead.
// ---------------------------------------------------------------------------
struct TileSmem {
  unsigned long long h[kWalkCells];     // elevations, final where eroded
  uint32_t acc[kWalkCells];             // drainage counts
  uint16_t list[kWalkCells];            // cells level by level
  uint8_t code[kWalkCells];
  unsigned long long rows[kRing][kWalkH];  // the cells of the last levels
  unsigned long long entry[kWalkH];     // cells that water of other tiles enters
  int end[kRing];                       // where the last levels end in the list
  int ready;                            // levels found (| kFinished: all)
  int done;                             // levels eroded
  int task, flag;
  int wide;                             // the level that all workers erode, or -1
};

__device__ __forceinline__ void st_volatile_i32(int *p, int v) {
  *reinterpret_cast<volatile int *>(p) = v;
}

struct Front {
  unsigned long long D[8];  // this lane's row: cells whose receiver lies in direction k
  unsigned long long flow;  // cells with a receiver
};

__device__ __forceinline__ void front_load(Front &f, const uint32_t *planes, int lane) {
  unsigned long long b[4];
#pragma unroll
  for (int p = 0; p < 4; p++) {
    const uint2 q = __ldcg(reinterpret_cast<const uint2 *>(planes + p * 64) + lane);
    b[p] = (unsigned long long)q.y << 32 | q.x;
  }
  f.flow = b[3];
#pragma unroll
  for (int k = 0; k < 8; k++)
    f.D[k] = b[3] & (k & 1 ? b[0] : ~b[0]) & (k & 2 ? b[1] : ~b[1]) & (k & 4 ? b[2] : ~b[2]);
}

// Donors in this lane's row of a set of cells given as the rows above, at and
// below (U, M, B), each with the cells left and right of the tile (bit 0 of
// xl, xr).
__device__ __forceinline__ unsigned long long donors_row(
    const Front &f, unsigned long long U, unsigned long long ul, unsigned long long ur,
    unsigned long long M, unsigned long long ml, unsigned long long mr, unsigned long long B,
    unsigned long long bl, unsigned long long br) {
  return (f.D[0] & (M << 1 | ml)) | (f.D[1] & (U << 1 | ul)) | (f.D[2] & U) |
         (f.D[3] & (U >> 1 | ur << 63)) | (f.D[4] & (M >> 1 | mr << 63)) |
         (f.D[5] & (B >> 1 | br << 63)) | (f.D[6] & B) | (f.D[7] & (B << 1 | bl));
}

// The donors of F inside the tile.
__device__ __forceinline__ unsigned long long front_next(const Front &f, unsigned long long F,
                                                         int lane) {
  unsigned long long up = __shfl_up_sync(kFull, F, 1), dn = __shfl_down_sync(kFull, F, 1);
  if (lane == 0) up = 0;
  if (lane == 31) dn = 0;
  return donors_row(f, up, 0, 0, F, 0, 0, dn, 0, 0);
}

// Appends the cells of the lanes' rows m to list from pos on; returns the end
// and, where asked for, the place of the lane's first.
__device__ __forceinline__ int front_emit(unsigned long long m, int lane, uint16_t *list, int pos,
                                          int *first = nullptr) {
  const int n = __popcll(m);
  int incl = n;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const int y = __shfl_up_sync(kFull, incl, s);
    if (lane >= s) incl += y;
  }
  const int total = __shfl_sync(kFull, incl, 31);
  if (first) *first = pos + incl - n;
  uint16_t *to = list + pos + incl - n;
  for (uint32_t w = (uint32_t)m; w; w &= w - 1) *to++ = (uint16_t)(64 * lane + __ffs(w) - 1);
  for (uint32_t w = (uint32_t)(m >> 32); w; w &= w - 1) *to++ = (uint16_t)(64 * lane + __ffs(w) + 31);
  return pos + total;
}

// The exits whose receivers are final: donors of the final cells just outside
// the tile. Relaxed loads, all in flight at once (each acquire would wait for
// its own, 700 clocks); a caller that goes on to read elevations fences first.
__device__ __forceinline__ unsigned long long ready_exits(const StepArgs &a, int t, const Tile &tl,
                                                          int W, int H, const Front &f, int lane) {
  const unsigned long long *done = a.tb.done;
  auto row = [&](bool there, int tile, int y) -> unsigned long long {
    return there ? ld_relaxed_u64(done + (size_t)tile * kWalkH + y) : 0ull;
  };
  const bool w = tl.x0 > 0, e = tl.x0 + kWalkW < W, n = tl.y0 > 0, so = tl.y0 + kWalkH < H;
  const bool top = lane == 0, bottom = lane == 31;
  // one row of each neighbour above or below, for the first and last lane
  const int tv = top ? t - tl.ntx : t + tl.ntx, yv = top ? kWalkH - 1 : 0;
  const bool there = (top && n) || (bottom && so);
  const unsigned long long l = row(w, t - 1, lane), r = row(e, t + 1, lane);
  const unsigned long long v = row(there, tv, yv), vl = row(there && w, tv - 1, yv),
                           vr = row(there && e, tv + 1, yv);
  const unsigned long long L = l >> 63, R = r & 1ull;
  unsigned long long lu = __shfl_up_sync(kFull, L, 1), ru = __shfl_up_sync(kFull, R, 1);
  unsigned long long ld = __shfl_down_sync(kFull, L, 1), rd = __shfl_down_sync(kFull, R, 1);
  if (top) {
    lu = vl >> 63;
    ru = vr & 1ull;
  }
  if (bottom) {
    ld = vl >> 63;
    rd = vr & 1ull;
  }
  return donors_row(f, top ? v : 0, lu, ru, 0, L, R, bottom ? v : 0, ld, rd);
}

// Changes whenever a tile gets further: the finished tiles, or cells, and the
// tiles' own reports in one word (one of each does not cancel).
__device__ __forceinline__ unsigned tiles_moved(const Ctl *ctl) {
  return (unsigned)ld_volatile_i32(&ctl->progress) * 0x10001u + (unsigned)ld_volatile_i32(&ctl->left);
}

// Queues tile u unless it is queued or at work already; then it runs again.
__device__ __forceinline__ void queue_push(const StepArgs &a, int u) {
  if (atomicOr(a.tb.state + u, kTileQueued | kTileAgain) & kTileQueued) return;
  __threadfence();  // what the tile's last block wrote, before its next one
  const unsigned at = atomicAdd(&a.ctl->qtail, 1u) % (unsigned)a.tb.n;
  // A tile is in the ring once at most, so the place is free, or its block
  // about to take the tile from it: bounded all the same.
  unsigned long long t0 = 0;
  for (unsigned n = 0; atomicCAS(a.tb.queue + at, 0, u + 1) != 0; ++n) {
    if (ld_volatile_i32(&a.ctl->err) != 0) return;
    if ((n & 63u) != 63u) continue;
    const unsigned long long now = globaltimer_ns();
    if (n == 63u) t0 = now;
    if (now - t0 > a.timeout_ns) {
      raise_err(a.ctl, FS_ERR_TIMEOUT, kPhaseBarrier);
      return;
    }
  }
}

// Queues the neighbours that drain into the newly final cells e of the lanes'
// rows (whole warp).
__device__ __forceinline__ void queue_neighbours(const StepArgs &a, int t, const Tile &tl, int W,
                                                 int H, unsigned long long e, int lane) {
  unsigned m = 0;
  const unsigned l = (unsigned)(e & 1ull), r = (unsigned)(e >> 63);
  if (l) m |= 1u << 3;
  if (r) m |= 1u << 5;
  if (lane == 0 && e) m |= 1u << 1 | l << 0 | r << 2;
  if (lane == 31 && e) m |= 1u << 7 | l << 6 | r << 8;
  m = __reduce_or_sync(kFull, m);
  if (lane < 9 && (m >> lane & 1u)) {
    const int dx = lane % 3 - 1, dy = lane / 3 - 1;
    const int x = tl.x0 + dx * kWalkW, y = tl.y0 + dy * kWalkH;
    if (x >= 0 && y >= 0 && x < W && y < H) queue_push(a, t + dy * tl.ntx + dx);
  }
  __syncwarp();
}

// Warp 0. F: the next level (kResident: level 1, the pits being level 0),
// claimed: cells found so far or final before, and on return all of
// them. Returns the list's end.
template <int MODE>
__device__ __forceinline__ int find_levels(const StepArgs &a, int t, const Tile &tl, int W, int H,
                                           TileSmem &s, const Front &f, unsigned long long F,
                                           unsigned long long &claimed, int pos, int lane) {
  int prod = 1, pub = MODE == kQueued ? 1 : 0;
  const unsigned long long entry = s.entry[lane];
  unsigned long long *own = a.tb.done + (size_t)t * kWalkH + lane;
  unsigned long long fin = MODE == kQueued ? claimed : 0;  // final and published, or about to be
  unsigned long long since = 0;                            // kQueued: final since the last publication
  unsigned long long t0 = 0;
  unsigned idle = 0;
  unsigned seen = 0;
  auto publish = [&]() {
    __threadfence();  // the elevations (the workers' barrier, then s.done) before the bits
    *reinterpret_cast<volatile unsigned long long *>(own) = fin;
    if (MODE == kQueued) {
      __threadfence();
      __syncwarp();
      queue_neighbours(a, t, tl, W, H, since & entry, lane);
    }
    since = 0;
  };
  for (;;) {
    const bool some = __any_sync(kFull, F != 0);
    const int dn = __shfl_sync(kFull, ld_volatile_i32(&s.done), 0);
    if (some && prod - dn < kLead) {
      s.rows[prod % kRing][lane] = F;
      pos = front_emit(F, lane, s.list, pos);
      if (lane == 0) s.end[prod % kRing] = pos;
      ++prod;
      __threadfence_block();
      __syncwarp();
      if (lane == 0) {
        st_volatile_i32(&s.ready, prod);
        if (prod % 16 == 0) atomicAdd(&a.ctl->progress, 1);
      }
      claimed |= F;
      F = front_next(f, F, lane);
      idle = 0;
    }
    if (dn > pub) {
      __threadfence_block();
      for (; pub < dn; ++pub) since |= s.rows[pub % kRing][lane];
      fin |= since;
      // kQueued: every few levels, since its publication looks for tiles to queue
      if (__any_sync(kFull, (since & entry) != 0) && (MODE == kResident || dn % kRing == 0)) publish();
    }
    if (!some || prod - dn >= 2) {
      const unsigned long long R = ready_exits(a, t, tl, W, H, f, lane) & ~(claimed | F);
      F |= R;
      const bool found = __any_sync(kFull, R != 0);
      if (found) __threadfence();  // the bits before the elevations
      if (!some && dn == prod && !found) {
        if (MODE == kQueued || !__any_sync(kFull, (f.flow & ~claimed) != 0)) break;
        // Waiting for the neighbours: bounded, while no tile gets further. A
        // tile counts as getting further with every 16th level, when it waits
        // again after some (here, where it costs nothing: told at each
        // publication, eroded 512^2 took 4% longer) and when it is finished.
        if ((++idle & 15u) == 0) {
          const unsigned long long now = globaltimer_ns();
          if (idle == 16 && lane == 0) atomicAdd(&a.ctl->progress, 1);
          const unsigned p = tiles_moved(a.ctl);
          if (idle == 16 || p != seen) {
            t0 = now;
            seen = p;
          }
          if (ld_volatile_i32(&a.ctl->err) != 0) break;
          if (now - t0 > a.timeout_ns) {
            if (lane == 0) raise_err(a.ctl, FS_ERR_TIMEOUT, kPhaseBarrier);
            break;
          }
        }
        __nanosleep(40);
      }
    }
  }
  if (MODE == kQueued) {
    for (; pub < prod; ++pub) since |= s.rows[pub % kRing][lane];
    fin |= since;
    publish();
  }
  __syncwarp();
  if (lane == 0) st_volatile_i32(&s.ready, prod | kFinished);
  return pos;
}

// One cell on its way to being eroded.
struct Cell {
  int c, rc;    // the cell, and its receiver's inside the tile (-1: outside)
  bool out;     // cells of other tiles drain into it: its elevation goes there
  uint64_t h0;  // uplifted elevation
  uint64_t hx;  // the receiver's, outside
  const unsigned long long *Tb;
  ulonglong2 fd;  // F, D
  uint64_t rn;    // -1/D
};

// The table record of drainage count k and direction dir.
template <int NMODE, int VAR>
__device__ __forceinline__ void cell_table(Cell &e, const RealDesc &d, uint32_t k, int dir) {
  e.Tb = reinterpret_cast<const unsigned long long *>(d.tab) + (size_t)k * kTabStride + 4 * (dir & 1);
  if (NMODE == kNOne && VAR != 2) {
    e.fd = __ldg(reinterpret_cast<const ulonglong2 *>(e.Tb));
    e.rn = __ldg(e.Tb + 3);
  } else {
    e.fd.x = __ldg(e.Tb);
  }
}

// The cell's final elevation from its receiver's (fastscape_RB.cpp:315-326).
template <int NMODE, int VAR>
__device__ __forceinline__ uint64_t cell_erode(const Cell &e, const Tolerance &tol, double neq,
                                               Ctl *ctl, uint64_t hn) {
  uint64_t h;
  if (NMODE == kNOne && VAR != 2) {
    h = erode_cell_n1<VAR == 1>(tol, ctl, e.Tb, TabN1{e.fd.x, e.fd.y, e.rn}, e.h0, hn);
  } else if (NMODE == kNTwo && VAR != 2) {
    h = erode_cell_n2<VAR == 1>(tol, neq, ctl, e.fd.x, e.h0, hn);
  } else {
    h = (uint64_t)__double_as_longlong(
        erode_cell<NMODE>(tol, neq, ctl, reinterpret_cast<const double *>(e.Tb),
                          __longlong_as_double(e.h0), __longlong_as_double(hn)));
  }
  if (((h >> 52) & 0x7FF) == 0x7FF) raise_err(ctl, FS_ERR_NONFINITE, kPhaseErode);  // Inf or NaN
  return h;
}

// The other warps. staged: the tile's elevations, counts and codes are in
// shared memory (kResident: always).
template <int NMODE, int VAR, int MODE, int WORKERS>
__device__ __forceinline__ void erode_levels(const StepArgs &a, int t, const Tile &tl,
                                             const RealDesc &d, TileSmem &s, bool staged) {
  constexpr bool kHelpers = WORKERS > kCore;
  const int wt = (int)threadIdx.x - 32;
  const int W = d.W;
  const uint64_t udt = (uint64_t)__double_as_longlong(d.u_dt);
  const Tolerance tol = d.tol;
  unsigned long long *gh = reinterpret_cast<unsigned long long *>(a.h + d.off);
  const int org = tl.y0 * W + tl.x0;
  auto grid_cell = [&](int c) { return org + (c >> 6) * W + (c & 63); };
  auto load = [&](int i, int hi) -> Cell {
    Cell e;
    e.c = -1;
    e.rc = -1;
    e.h0 = e.hx = 0;
    e.out = MODE == kQueued;
    if (i < hi) {
      e.c = s.list[i];
      if (MODE == kResident) e.out = s.entry[e.c >> 6] >> (e.c & 63) & 1ull;
      int code;
      uint32_t k;
      uint64_t h;
      if (MODE != kQueued || staged) {
        code = s.code[e.c];
        k = s.acc[e.c];
        h = s.h[e.c];
      } else {
        const int g = grid_cell(e.c);
        code = __ldg(a.tb.code + (size_t)t * kWalkCells + e.c);
        k = __ldcg(a.tb.count + d.off + g);
        h = __ldcg(gh + g);
      }
      const int dir = code & 7;
      if (code >= kCodeExit) e.hx = __ldcg(gh + grid_cell(e.c) + nbr_off(dir, W));
      else e.rc = e.c + tile_off(dir);
      cell_table<NMODE, VAR>(e, d, k, dir);
      e.h0 = h;  // to be uplifted
    }
    return e;
  };
  auto turn = [&](int L) -> int {  // place among the level's workers
    const int k = (wt >> 5) - L % (kCore / 32);
    return 32 * (k < 0 ? k + kCore / 32 : k) + (wt & 31);
  };
  auto erode = [&](const Cell &e) {
    const uint64_t hn = e.rc >= 0 ? s.h[e.rc] : e.hx;
    const uint64_t h = cell_erode<NMODE, VAR>(e, tol, a.neq, a.ctl, hn);
    s.h[e.c] = h;
    if (e.out) gh[grid_cell(e.c)] = h;
  };
  auto erode_from = [&](int i, int hi, int step) {
    for (; i < hi; i += step) {
      Cell e = load(i, hi);
      e.h0 = uplift_bits(e.h0, udt);
      erode(e);
    }
  };
  if (kHelpers && wt >= kCore) {  // wide levels only; asleep at the barrier between them
    for (;;) {
      group_sync(2, WORKERS);
      const int L = s.wide;
      if (L < 0) return;
      erode_from(s.end[(L - 1) % kRing] + wt, s.end[L % kRing], WORKERS);
      group_sync(2, WORKERS);
    }
  }
  // nx: this thread's first cell of the level, loaded during the level before
  // (first == L). The warps take turns: level L's first 32 cells, on deep
  // ground often all of them, are warp L % 3's, which has loaded and uplifted
  // them while another warp eroded the level before.
  int first = -1;
  Cell nx;
  for (int L = MODE == kQueued ? 1 : 0;; ++L) {
    int ready;
    for (unsigned n = 0; (ready = ld_volatile_i32(&s.ready)) <= L; ++n)
      if (n > 2) __nanosleep(50);
    if ((ready &= ~kFinished) <= L) {
      if (kHelpers) {
        if (wt == 0) s.wide = -1;
        group_sync(2, WORKERS);
      }
      return;
    }
    __threadfence_block();
    const int lo = L ? s.end[(L - 1) % kRing] : 0, hi = s.end[L % kRing];
    const int at = lo + turn(L);
    Cell e = nx;
    if (first != L && L) {
      e = load(at, hi);
      if (e.c >= 0) e.h0 = uplift_bits(e.h0, udt);
    }
    const bool more = ready > L + 1;
    if (more) nx = load(hi + turn(L + 1), s.end[(L + 1) % kRing]);
    const bool wide = kHelpers && L && hi - lo > 2 * kCore;
    if (wide) {
      if (wt == 0) s.wide = L;
      group_sync(2, WORKERS);
    }
    if (MODE != kQueued && L == 0) {
      // level 0, of which the pits rise with the land (fastscape_RB.cpp:291-295)
      for (int i = wt; i < hi; i += kCore) {
        const int c = s.list[i];
        const uint64_t h = fadd_bits(s.h[c], udt);
        s.h[c] = h;
        if (MODE == kResident && (s.entry[c >> 6] >> (c & 63) & 1ull)) gh[grid_cell(c)] = h;
      }
    } else if (e.c >= 0) {
      erode(e);
      const int step = wide ? WORKERS : kCore;
      erode_from(at + step, hi, step);
    }
    if (more) {
      first = L + 1;
      if (nx.c >= 0) nx.h0 = uplift_bits(nx.h0, udt);
    }
    if (wide) group_sync(2, WORKERS);
    else group_sync(1, kCore);
    if (wt == 0) {
      __threadfence_block();
      st_volatile_i32(&s.done, L + 1);
    }
  }
}

// The tile's drainage counts: those of its own cells, and the water from
// other tiles along its way (block-wide; ends with a barrier).
__device__ __forceinline__ void tile_counts(const StepArgs &a, int t, uint32_t *acc, uint8_t *code,
                                            unsigned long long *entry) {
  const int tid = threadIdx.x, n = blockDim.x;
  for (int i = tid; i < kWalkCells / 8; i += n) {
    const uint4 q = __ldcg(reinterpret_cast<const uint4 *>(a.tb.local + (size_t)t * kWalkCells) + i);
    uint4 *to = reinterpret_cast<uint4 *>(acc + 8 * i);
    to[0] = make_uint4(q.x & 0xFFFFu, q.x >> 16, q.y & 0xFFFFu, q.y >> 16);
    to[1] = make_uint4(q.z & 0xFFFFu, q.z >> 16, q.w & 0xFFFFu, q.w >> 16);
  }
  for (int i = tid; i < kWalkCells / 16; i += n)
    reinterpret_cast<uint4 *>(code)[i] =
        __ldcg(reinterpret_cast<const uint4 *>(a.tb.code + (size_t)t * kWalkCells) + i);
  if (entry && tid < kWalkH) entry[tid] = 0;
  uint32_t in[2];
#pragma unroll
  for (int j = 0; j < 2; j++)
    in[j] = tid + j * n < kSlots ? __ldcg(a.tb.inflow + (size_t)t * kSlots + tid + j * n) : 0u;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 2; j++)
    if (in[j]) {
      int c = slot_cell(tid + j * n);
      if (entry) atomicOr(&entry[c >> 6], 1ull << (c & 63));
      for (int k = 0; k < kWalkCells; k++) {
        atomicAdd(&acc[c], in[j]);
        const int dir = code[c];
        if (dir >= 8) break;
        c += tile_off(dir);
      }
    }
  cp_async_wait();
  __syncthreads();
}

__global__ void __launch_bounds__(kWalkThreads) k_tile_counts(StepArgs a) {
  if (stopped(a.ctl)) return;
  __shared__ __align__(16) uint32_t s_acc[kWalkCells];
  __shared__ __align__(16) uint8_t s_code[kWalkCells];
  const int t = tile_of(a, blockIdx.x);
  const Tile tl = a.tb.tiles[t];
  const RealDesc &d = a.tb.desc[tl.r];
  tile_counts(a, t, s_acc, s_code, nullptr);
  const int wcells = min(kWalkW, d.W - tl.x0), hrows = min(kWalkH, d.H - tl.y0);
  for (int y = threadIdx.x >> 5; y < hrows; y += kWalkThreads / 32)
    for (int x = threadIdx.x & 31; x < wcells; x += 32)
      a.tb.count[d.off + (size_t)(tl.y0 + y) * d.W + tl.x0 + x] = s_acc[y * 64 + x];
}

// The tile's elevations into shared memory (asynchronous; tile_counts waits).
template <int THREADS>
__device__ __forceinline__ void tile_stage(const StepArgs &a, const Tile &tl, const RealDesc &d,
                                           unsigned long long *h) {
  const unsigned long long *gh = reinterpret_cast<const unsigned long long *>(a.h + d.off);
  const int x = threadIdx.x & 63, hrows = min(kWalkH, d.H - tl.y0);
  if (tl.x0 + x < d.W) {
    const unsigned long long *p = gh + (size_t)(tl.y0 + (threadIdx.x >> 6)) * d.W + tl.x0 + x;
    for (int y = threadIdx.x >> 6; y < hrows; y += THREADS / 64, p += THREADS / 64 * d.W)
      cp_async8(h + y * 64 + x, p);
  }
}

// And back.
template <int THREADS>
__device__ __forceinline__ void tile_store(const StepArgs &a, const Tile &tl, const RealDesc &d,
                                           const unsigned long long *h) {
  unsigned long long *gh = reinterpret_cast<unsigned long long *>(a.h + d.off);
  const int x = threadIdx.x & 63, hrows = min(kWalkH, d.H - tl.y0);
  if (tl.x0 + x < d.W) {
    unsigned long long *p = gh + (size_t)(tl.y0 + (threadIdx.x >> 6)) * d.W + tl.x0 + x;
    for (int y = threadIdx.x >> 6; y < hrows; y += THREADS / 64, p += THREADS / 64 * d.W)
      *p = h[y * 64 + x];
  }
}

// Warp 0: level 0, the cells without a receiver (this lane's row), and of
// these the pits, the interior ones, which alone rise with the land
// (fastscape_RB.cpp:291-295).
__device__ __forceinline__ unsigned long long root_row(const Tile &tl, int W, int H,
                                                       const Front &f, int lane,
                                                       unsigned long long *pits) {
  const int wcells = min(kWalkW, W - tl.x0), hrows = min(kWalkH, H - tl.y0);
  const unsigned long long cols = wcells == 64 ? ~0ull : (1ull << wcells) - 1ull;
  unsigned long long inner = cols;  // columns 2 .. W-3 of the grid
  if (tl.x0 == 0) inner &= ~3ull;
  if (W - 2 - tl.x0 < 64) inner &= W - 2 - tl.x0 > 0 ? (1ull << (W - 2 - tl.x0)) - 1ull : 0ull;
  const int gy = tl.y0 + lane;
  const unsigned long long roots = lane < hrows ? cols & ~f.flow : 0ull;
  *pits = gy >= 2 && gy < H - 2 ? roots & inner : 0ull;
  return roots;
}

template <int NMODE, int VAR, int T>
__global__ void __launch_bounds__(T, 768 / T) k_tile_resident(StepArgs a) {
  if (stopped(a.ctl)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TileSmem &s = *reinterpret_cast<TileSmem *>(smem_raw);
  const int t = tile_of(a, blockIdx.x);
  const Tile tl = a.tb.tiles[t];
  const RealDesc &d = a.tb.desc[tl.r];
  const int lane = threadIdx.x & 31;
  tile_stage<T>(a, tl, d, s.h);
  if (threadIdx.x == 0) s.ready = s.done = 0;
  tile_counts(a, t, s.acc, s.code, s.entry);
  if (threadIdx.x < 32) {
    Front f;
    front_load(f, a.tb.planes + (size_t)t * 256, lane);
    unsigned long long pits;
    unsigned long long final = root_row(tl, d.W, d.H, f, lane, &pits);
    const int pos = front_emit(pits, lane, s.list, 0);
    if (lane == 0) s.end[0] = pos;
    s.rows[0][lane] = final;
    __threadfence_block();
    __syncwarp();
    if (lane == 0) st_volatile_i32(&s.ready, 1);
    find_levels<kResident>(a, t, tl, d.W, d.H, s, f, front_next(f, final, lane), final, pos, lane);
  } else {
    erode_levels<NMODE, VAR, kResident, T - 32>(a, t, tl, d, s, true);
  }
  __syncthreads();
  tile_store<T>(a, tl, d, s.h);
  if (threadIdx.x == 0 && atomicAdd(&a.ctl->left, 1) == (int)gridDim.x - 1)
    atomicAdd(&a.ctl->steps_done, 1);
}

// Grids of more tiles than fit the GPU. Most cells are eroded here (96% of
// young ground). The issue slots bound it, then the FP64 pipe (four
// operations a cell): six blocks fit an SM, so that the barriers of one and
// the single warp that finds levels are covered by the others. Levels 1 and
// 2, four fifths of young ground, are listed by all warps, a word of 32 cells
// at a time.
struct RootedSmem {
  unsigned long long h[kWalkCells];
  uint32_t acc[kWalkCells];
  uint16_t list[kWalkCells];
  uint8_t code[kWalkCells];
  uint32_t words[3][2 * kWalkH];  // pits, level 1, level 2
  uint16_t base[2][2 * kWalkH];   // where each word's cells go in the list
  int end[4];
  int left;
};

// The cells of a tile that k_tile_rooted leaves to k_tile_pull (at most
// kPullMost, in row order): the cell with its direction in bits 11 to 13, its
// uplifted elevation and count, where each row's begin, and afterwards which
// are done. They take the place of links and sinks, spent by then.
struct TileRest {
  uint16_t *cell;            // [kPullMost]
  unsigned long long *h0;    // [kPullMost]
  uint32_t *count;           // [kPullMost]
  uint16_t *row;             // [kWalkH]
  uint32_t *pulled;          // [kPullMost / 32]
};

__device__ __forceinline__ TileRest tile_rest(const StepArgs &a, int t) {
  static_assert(kPullMost * 2 <= kSlots * 4 && kPullMost * 12 <= 2 * kSlots * 8 &&
                    kPullMost / 8 + kWalkH * 2 <= kSlots * 4,
                "the tile's spent arrays hold its rest");
  TileRest r;
  r.cell = reinterpret_cast<uint16_t *>(a.tb.start + (size_t)t * kSlots);
  r.h0 = a.tb.sink + (size_t)t * (2 * kSlots);
  r.count = reinterpret_cast<uint32_t *>(r.h0 + kPullMost);
  r.pulled = a.tb.link + (size_t)t * kSlots;
  r.row = reinterpret_cast<uint16_t *>(r.pulled + kPullMost / 32);
  return r;
}

template <int NMODE, int VAR>
__global__ void __launch_bounds__(kRootedThreads, 6) k_tile_rooted(StepArgs a) {
  if (stopped(a.ctl)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RootedSmem &s = *reinterpret_cast<RootedSmem *>(smem_raw);
  const int t = tile_of(a, blockIdx.x);
  const Tile tl = a.tb.tiles[t];
  const RealDesc &d = a.tb.desc[tl.r];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, wt = (int)threadIdx.x - 32;
  constexpr int kWarps = kRootedThreads / 32, kErode = kRootedThreads - 32;
  constexpr bool kRounds = NMODE != kNOne;  // what is left is k_tile_front's
  const uint64_t udt = (uint64_t)__double_as_longlong(d.u_dt);
  const Tolerance tol = d.tol;
  tile_stage<kRootedThreads>(a, tl, d, s.h);
  Front f;
  unsigned long long F = 0, F1 = 0, final = 0;  // the last level found, the one before, all
  int pos = 0;
  if (wid == 0) {  // levels 0 to 2
    front_load(f, a.tb.planes + (size_t)t * 256, lane);
    unsigned long long pits;
    F = final = root_row(tl, d.W, d.H, f, lane, &pits);
    reinterpret_cast<unsigned long long *>(s.words[0])[lane] = pits;
#pragma unroll
    for (int q = 0; q < 2; q++) {
      if (kRounds) F1 = F;
      F = front_next(f, F, lane);
      final |= F;
      const int nl = __popc((uint32_t)F), n = nl + __popc((uint32_t)(F >> 32));
      int incl = n;
#pragma unroll
      for (int k = 1; k < 32; k <<= 1) {
        const int v = __shfl_up_sync(kFull, incl, k);
        if (lane >= k) incl += v;
      }
      reinterpret_cast<unsigned long long *>(s.words[q + 1])[lane] = F;
      s.base[q][2 * lane] = (uint16_t)(pos + incl - n);
      s.base[q][2 * lane + 1] = (uint16_t)(pos + incl - n + nl);
      pos += __shfl_sync(kFull, incl, 31);
      if (lane == 0) s.end[q + 1] = pos;
    }
    if (lane == 0) s.end[0] = 0;
  }
  tile_counts(a, t, s.acc, s.code, nullptr);
  for (int w = wid; w < 2 * kWalkH; w += kWarps) {
    const uint32_t p = s.words[0][w];
    if (p >> lane & 1u) {  // the pits' uplift
      unsigned long long &h = s.h[32 * w + lane];
      h = fadd_bits(h, udt);
    }
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const uint32_t m = s.words[q + 1][w];
      if (m >> lane & 1u)
        s.list[s.base[q][w] + __popc(m & ((1u << lane) - 1u))] = (uint16_t)(32 * w + lane);
    }
  }
  __syncthreads();
  auto load = [&](int i, int hi) -> Cell {
    Cell e;
    e.c = e.rc = 0;
    if (i < hi) {
      e.c = s.list[i];
      const int dir = s.code[e.c];
      e.rc = e.c + tile_off(dir);
      cell_table<NMODE, VAR>(e, d, s.acc[e.c], dir);
      e.h0 = uplift_bits(s.h[e.c], udt);
    }
    return e;
  };
  Cell nx;
  if (wid) nx = load(wt, s.end[1]);
  for (int L = 1;; ++L) {
    const int lo = s.end[(L - 1) & 3], hi = s.end[L & 3], hi2 = s.end[(L + 1) & 3];
    if (lo == hi) break;
    if (kRounds && (hi - lo < (NMODE == kNTwo ? kRootedFewTwo : kRootedFewGeneral) ||
                    (NMODE == kNGeneral && gridDim.x < kRootedWaves))) {
      // k_tile_front's from here on
      if (wid == 0) final &= ~(F | F1);
      break;
    }
    if (wid == 0) {  // level L + 2
      if (kRounds) F1 = F;
      F = front_next(f, F, lane);
      final |= F;
      pos = front_emit(F, lane, s.list, pos);
      if (lane == 0) s.end[(L + 2) & 3] = pos;
    } else {
      for (int i = lo + wt; i < hi; i += kErode) {
        const Cell e = nx;
        nx = load(i + kErode, hi);
        s.h[e.c] = cell_erode<NMODE, VAR>(e, tol, a.neq, a.ctl, s.h[e.rc]);
      }
      nx = load(hi + wt, hi2);
    }
    __syncthreads();
  }
  tile_store<kRootedThreads>(a, tl, d, s.h);
  // The cells of trees that leave the tile: a few for k_tile_pull, many for
  // the queue, or all for k_tile_front. Only their counts go to memory (the
  // others': k_tile_counts, when a caller asks).
  const TileRest rest = tile_rest(a, t);
  if (wid == 0) {
    a.tb.done[(size_t)t * kWalkH + lane] = final;
    const unsigned long long rows = f.flow & ~final;
    int at;
    const int left = front_emit(rows, lane, s.list, 0, &at);
    if (!kRounds) rest.row[lane] = (uint16_t)at;
    if (lane == 0) {
      const bool pull = kRounds || left <= kPullMost;
      s.left = left;
      a.tb.nstart[t] = pull ? left : 0;
      if (kRounds && left) atomicAdd(&a.ctl->left, left);
      if (!pull) {
        atomicAdd(&a.ctl->left, left);
        a.tb.state[t] = kTileQueued;
        a.tb.queue[atomicAdd(&a.ctl->qtail, 1u)] = t + 1;
      }
    }
  }
  __syncthreads();
  const int left = s.left;
  for (int i = threadIdx.x; i < left; i += kRootedThreads) {
    const int c = s.list[i];
    a.tb.count[d.off + (size_t)(tl.y0 + (c >> 6)) * d.W + tl.x0 + (c & 63)] = s.acc[c];
    if (!kRounds && left <= kPullMost) {
      rest.cell[i] = (uint16_t)(c | (s.code[c] & 7) << 11);
      rest.h0[i] = uplift_bits(s.h[c], udt);
      rest.count[i] = s.acc[c];
    }
  }
}

// Cells whose receivers lead into another tile within a few steps -- nearly
// all that are left on young ground, where they are one to four steps from a
// final cell. A thread takes one: it follows the receivers up to a final cell
// and erodes the path back down, its own cell last. A cell on several paths
// is eroded as often (1.3 times on average), by the same operations on the
// same operands; nothing waits, since the paths' uplifted elevations lie
// aside and the grid's are read where they were final before. Longer paths
// are k_tile_queue's. Waiting for gathers bounds it, so 14 blocks share an SM
// (48 registers, 40 bytes spilled; with the kernels after it 354 us of a
// 10000^2 timestep at ten blocks, 317 at 12, 278 at 14, 330 at 16).
template <int NMODE, int VAR>
__global__ void __launch_bounds__(kPullThreads, 14) k_tile_pull(StepArgs a) {
  if (stopped(a.ctl)) return;
  __shared__ unsigned s_path[kPullDepth][kPullThreads];  // tile * kPullMost + index
  __shared__ int s_fail;
  const int lane = threadIdx.x & 31;
  const int t = tile_of(a, blockIdx.x);
  const int n = a.tb.nstart[t];
  if (n == 0) return;
  const Tile tl = a.tb.tiles[t];
  const RealDesc &d = a.tb.desc[tl.r];
  const int W = d.W;
  const Tolerance tol = d.tol;
  unsigned long long *gh = reinterpret_cast<unsigned long long *>(a.h + d.off);
  if (threadIdx.x == 0) s_fail = 0;
  __syncthreads();
  for (int i = threadIdx.x; i - lane < n; i += kPullThreads) {
    bool ok = false;
    if (i < n) {
      int u = t, at = i, x, y, g0 = 0, depth = 0;
      for (;;) {
        const int e = tile_rest(a, u).cell[at];
        const int ux = u == t ? tl.x0 : x & ~(kWalkW - 1), uy = u == t ? tl.y0 : y & ~(kWalkH - 1);
        x = ux + (e & 63);
        y = uy + (e >> 6 & (kWalkH - 1));
        if (depth == 0) g0 = y * W + x;
        s_path[depth++][threadIdx.x] = (unsigned)u * kPullMost + at;
        x += dir_dx(e >> 11);
        y += dir_dy(e >> 11);
        u = d.tile0 + (y / kWalkH) * tl.ntx + x / kWalkW;
        const unsigned long long done = __ldg(a.tb.done + (size_t)u * kWalkH + y % kWalkH);
        ok = done >> (x % kWalkW) & 1ull;
        if (ok || depth == kPullDepth || a.tb.nstart[u] == 0) break;  // 0: the queue's tile
        // the receiver's place in its tile's rest
        const unsigned long long flow =
            __ldg(reinterpret_cast<const unsigned long long *>(a.tb.planes + (size_t)u * 256 + 192) +
                  y % kWalkH);
        at = tile_rest(a, u).row[y % kWalkH] +
             __popcll(flow & ~done & ((1ull << (x % kWalkW)) - 1ull));
      }
      if (ok) {
        uint64_t h = __ldcg(gh + (size_t)y * W + x);
        while (depth > 0) {
          const unsigned p = s_path[--depth][threadIdx.x];
          const TileRest rest = tile_rest(a, (int)(p / kPullMost));
          const int q = (int)(p % kPullMost);
          Cell e;
          e.h0 = rest.h0[q];
          cell_table<NMODE, VAR>(e, d, rest.count[q], rest.cell[q] >> 11);
          h = cell_erode<NMODE, VAR>(e, tol, a.neq, a.ctl, h);
        }
        gh[g0] = h;
      }
    }
    const unsigned m = __ballot_sync(kFull, ok);
    if (lane == 0) {
      tile_rest(a, t).pulled[i / 32] = m;
      const int fail = min(n - i, 32) - __popc(m);
      if (fail) atomicAdd(&s_fail, fail);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_fail) {
    atomicAdd(&a.ctl->left, s_fail);
    a.tb.state[t] = kTileQueued;
    a.tb.queue[atomicAdd(&a.ctl->qtail, 1u)] = t + 1;
  }
}

// Marks the cells that k_tile_pull finished, if the queue is to go on from
// them.
__global__ void __launch_bounds__(256) k_tile_mark(StepArgs a) {
  if (stopped(a.ctl) ||
      ld_volatile_i32(reinterpret_cast<const int *>(&a.ctl->qtail)) == 0)
    return;
  const int lane = threadIdx.x & 31;
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= a.tb.n) return;
  const int t = tile_of(a, w);
  const int n = a.tb.nstart[t];
  const TileRest rest = tile_rest(a, t);
  for (int i = lane; i < n; i += 32)
    if (rest.pulled[i / 32] >> (i & 31) & 1u) {
      const int c = rest.cell[i] & (kWalkCells - 1);
      atomicOr(a.tb.done + (size_t)t * kWalkH + (c >> 6), 1ull << (c & 63));
    }
}

// ---------------------------------------------------------------------------
// 4. The queue of tiles with unfinished cells, for grids of more tiles than
// fit the GPU. A tile is in the ring once at most; a block takes the next one,
// erodes what has become ready and queues the neighbours that wait for cells
// it finished. No block waits for a tile, only for the ring, so the order does
// not matter. A tile with many unfinished cells is staged like k_tile_resident's;
// of one with few (young ground: 80 of 2048) only those are gathered.
// ---------------------------------------------------------------------------

// The next tile, or -1 when every cell is final (one thread).
__device__ int queue_pop(const StepArgs &a) {
  Ctl *ctl = a.ctl;
  int32_t *at = a.tb.queue + atomicAdd(&ctl->qhead, 1u) % (unsigned)a.tb.n;
  unsigned long long t0 = globaltimer_ns();
  unsigned seen = 0;
  for (unsigned n = 0;; ++n) {
    const int v = ld_volatile_i32(at);
    if (v > 0 && atomicCAS(at, v, 0) == v) {
      __threadfence();
      return v - 1;
    }
    if (ld_volatile_i32(&ctl->left) == 0 || ld_volatile_i32(&ctl->err) != 0) return -1;
    if ((n & 63u) == 63u) {
      const unsigned long long now = globaltimer_ns();
      const unsigned p = tiles_moved(ctl);
      if (p != seen) {  // some tile got further
        seen = p;
        t0 = now;
      }
      if (now - t0 > a.timeout_ns) {
        raise_err(ctl, FS_ERR_TIMEOUT, kPhaseBarrier);
        return -1;
      }
    }
    __nanosleep(100);
  }
}

template <int NMODE, int VAR>
__global__ void __launch_bounds__(kWalkThreads, 7) k_tile_queue(StepArgs a) {
  Ctl *ctl = a.ctl;
  if (stopped(ctl)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TileSmem &s = *reinterpret_cast<TileSmem *>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  constexpr int kWarps = kWalkThreads / 32;
  // an empty queue stays empty: nothing is left
  if (blockIdx.x == 0 && tid == 0 && ld_volatile_i32(reinterpret_cast<const int *>(&ctl->qtail)) == 0)
    atomicAdd(&ctl->steps_done, 1);
  int again = 0;
  for (;;) {
    if (tid == 0 && !again) s.task = queue_pop(a);
    __syncthreads();
    const int t = s.task;
    if (t < 0) return;
    const Tile tl = a.tb.tiles[t];
    const RealDesc &d = a.tb.desc[tl.r];
    const int W = d.W, H = d.H;
    const unsigned long long *gh = reinterpret_cast<const unsigned long long *>(a.h + d.off);
    Front f;
    unsigned long long F = 0, own = 0;
    if (wid == 0) {
      if (lane == 0) atomicAnd(a.tb.state + t, ~kTileAgain);
      __threadfence();
      s.entry[lane] = 0;
      __syncwarp();
      front_load(f, a.tb.planes + (size_t)t * 256, lane);
      own = ld_relaxed_u64(a.tb.done + (size_t)t * kWalkH + lane);
      F = ready_exits(a, t, tl, W, H, f, lane) & ~own;
      __threadfence();  // the bits before the elevations
      // k_tile_pull may have finished a tree's lower part: go on above it
      const unsigned long long above = front_next(f, own, lane) & ~own;
      F |= above;
      for (int i = lane; i < kSlots; i += 32)
        if (__ldcg(a.tb.inflow + (size_t)t * kSlots + i)) {
          const int c = slot_cell(i);
          atomicOr(&s.entry[c >> 6], 1ull << (c & 63));
        }
      const int left = (int)__reduce_add_sync(kFull, (unsigned)__popcll(f.flow & ~own));
      const bool any = __any_sync(kFull, F != 0), staged = __any_sync(kFull, above != 0);
      if (lane == 0) {
        s.flag = !any ? 0 : staged || left > kStageFrom ? 2 : 1;
        s.ready = s.done = 1;
        s.end[0] = 0;
      }
    }
    __syncthreads();
    const int flag = s.flag;
    if (flag == 2) {
      const int wcells = min(kWalkW, W - tl.x0), hrows = min(kWalkH, H - tl.y0);
      for (int y = wid; y < hrows; y += kWarps)
        for (int x = lane; x < wcells; x += 32) {
          const size_t g = (size_t)(tl.y0 + y) * W + tl.x0 + x;
          cp_async8(&s.h[y * 64 + x], gh + g);
          s.acc[y * 64 + x] = __ldcg(a.tb.count + d.off + g);
        }
      for (int i = tid; i < kWalkCells / 16; i += kWalkThreads)
        reinterpret_cast<uint4 *>(s.code)[i] =
            __ldcg(reinterpret_cast<const uint4 *>(a.tb.code + (size_t)t * kWalkCells) + i);
      cp_async_wait();
      __syncthreads();
    }
    int n = 0;
    if (flag) {
      if (wid == 0) n = find_levels<kQueued>(a, t, tl, W, H, s, f, F, own, 0, lane);
      else erode_levels<NMODE, VAR, kQueued, kWalkThreads - 32>(a, t, tl, d, s, flag == 2);
    }
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      // queued again meanwhile: once more
      s.flag = atomicCAS(a.tb.state + t, (int)kTileQueued, 0) != kTileQueued;
      if (n && atomicAdd(&ctl->left, -n) == n) atomicAdd(&ctl->steps_done, 1);
    }
    __syncthreads();
    again = s.flag;
  }
}

// ---------------------------------------------------------------------------
// 5. Rounds of the whole GPU, where many cells are left or a cell takes long
// (n != 1): the cells whose receivers are final, then their donors, and so on,
// from one list that grows. Full warps are what counts there. k_tile_pull's lanes
// follow paths of their own and erode shared cells again (10000^2 with n = 1.5,
// 12 levels: 7.1 ms for 4% of the cells, 1.7 in rounds), and a tile from the
// queue is visited for few ready cells at a time. A round lasts as long as its
// slowest cell and a barrier, 20 us with n = 2, so the narrow rounds of long paths
// are left to k_tile_queue, whose tiles do not wait for one another's.
// ---------------------------------------------------------------------------
template <int NMODE, int VAR>
__global__ void __launch_bounds__(kFrontThreads, 2) k_tile_front(StepArgs a) {
  Ctl *ctl = a.ctl;
  if (stopped(ctl)) return;
  const int lane = threadIdx.x & 31;
  const int warp = (int)(blockIdx.x * kFrontThreads + threadIdx.x) >> 5;
  const int warps = (int)gridDim.x * (kFrontThreads / 32);
  const int all = ld_volatile_i32(&ctl->left);  // before the first barrier: written after it
  if (NMODE == kNOne && all < kFrontCells) return;
  // the list: cells numbered in their tile, and tiles
  int32_t *cell = a.amb, *tile = a.amb_r;
  // places for n entries of this lane (whole warps)
  auto places = [&](unsigned *count, int n) -> int {
    int incl = n;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const int v = __shfl_up_sync(kFull, incl, s);
      if (lane >= s) incl += v;
    }
    int at = 0;
    if (lane == 31 && incl) at = (int)atomicAdd(count, (unsigned)incl);
    return __shfl_sync(kFull, at, 31) + incl - n;
  };
  for (int w = warp; w < a.tb.n; w += warps) {
    const int t = tile_of(a, w);
    if (NMODE != kNOne && a.tb.nstart[t] == 0) continue;  // nothing left
    const Tile tl = a.tb.tiles[t];
    const RealDesc &d = a.tb.desc[tl.r];
    Front f;
    front_load(f, a.tb.planes + (size_t)t * 256, lane);
    const unsigned long long own = a.tb.done[(size_t)t * kWalkH + lane];
    unsigned long long F =
        (ready_exits(a, t, tl, d.W, d.H, f, lane) | front_next(f, own, lane)) & ~own;
    int at = places(&ctl->front[0], __popcll(F));
    for (; F; F &= F - 1, ++at) {
      cell[at] = 64 * lane + __ffsll((long long)F) - 1;
      tile[at] = t;
    }
  }
  unsigned epoch = 0;
  int lo = 0;
  for (unsigned r = 0;; ++r) {
    if (!grid_barrier(ctl, epoch, a.timeout_ns)) return;
    const int n = ld_volatile_i32(reinterpret_cast<const int *>(&ctl->front[r % 3]));
    if (n == 0 || (n < 32 * warps && all - lo > kFrontRounds * n)) break;
    unsigned *next = &ctl->front[(r + 1) % 3];
    if (blockIdx.x == 0 && threadIdx.x == 0) ctl->front[(r + 2) % 3] = 0;
    const int hi = lo + n;
    for (int i = lo + 32 * warp; i < hi; i += 32 * warps) {
      unsigned donors = 0;
      int c = 0, t = 0;
      Tile tl;
      if (i + lane < hi) {
        c = __ldcg(cell + i + lane);
        t = __ldcg(tile + i + lane);
        tl = a.tb.tiles[t];
        const RealDesc &d = a.tb.desc[tl.r];
        const int g = (tl.y0 + (c >> 6)) * d.W + tl.x0 + (c & 63);
        const int8_t *rec = a.rec + d.off + g;
        unsigned long long *h = reinterpret_cast<unsigned long long *>(a.h + d.off) + g;
        const int dir = __ldg(rec);
        const uint64_t h0 = __ldcg(h), hn = __ldcg(h + nbr_off(dir, d.W));
        Cell e;
        cell_table<NMODE, VAR>(e, d, __ldcg(a.tb.count + d.off + g), dir);
#pragma unroll
        for (int k = 0; k < 8; k++)
          if (__ldg(rec + nbr_off(k, d.W)) == ((k + 4) & 7)) donors |= 1u << k;
        e.h0 = uplift_bits(h0, (uint64_t)__double_as_longlong(d.u_dt));
        *h = cell_erode<NMODE, VAR>(e, d.tol, a.neq, ctl, hn);
      }
      int at = hi + places(next, __popc(donors));
      for (; donors; donors &= donors - 1, ++at) {
        const int k = __ffs(donors) - 1;
        const int x = (c & 63) + dir_dx(k), y = (c >> 6) + dir_dy(k);
        cell[at] = (y & (kWalkH - 1)) << 6 | (x & (kWalkW - 1));
        tile[at] = t + (y >> 5) * tl.ntx + (x >> 6);
      }
    }
    lo = hi;
  }
  // For the queue, in place of what k_tile_rooted and k_tile_pull put there:
  // what is final, and the tiles with cells left.
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctl->left = all - lo;
    ctl->qtail = 0;
  }
  for (int i = 32 * warp + lane; i < a.tb.n; i += 32 * warps) a.tb.queue[i] = 0;
  if (lo == all) return;
  for (int i = 32 * warp + lane; i < lo; i += 32 * warps) {
    const int c = __ldcg(cell + i);
    atomicOr(a.tb.done + (size_t)__ldcg(tile + i) * kWalkH + (c >> 6), 1ull << (c & 63));
  }
  if (!grid_barrier(ctl, epoch, a.timeout_ns)) return;
  for (int w = warp; w < a.tb.n; w += warps) {
    const int t = tile_of(a, w);
    const unsigned long long flow =
        __ldg(reinterpret_cast<const unsigned long long *>(a.tb.planes + (size_t)t * 256 + 192) + lane);
    if (!__any_sync(kFull, (flow & ~ld_relaxed_u64(a.tb.done + (size_t)t * kWalkH + lane)) != 0))
      continue;
    if (lane == 0) {
      a.tb.state[t] = kTileQueued;
      a.tb.queue[atomicAdd(&ctl->qtail, 1u)] = t + 1;
    }
  }
}

enum Kernel { kKernelRooted, kKernelPull, kKernelQueue, kKernelFront, kKernelResident };  // + width

template <int NMODE, int VAR>
const void *kernel_of_nv(int k) {
  if constexpr (NMODE == kNOne)
    if (k == kKernelPull) return reinterpret_cast<const void *>(&k_tile_pull<NMODE, VAR>);
  switch (k) {
    case kKernelFront: return reinterpret_cast<const void *>(&k_tile_front<NMODE, VAR>);
    case kKernelQueue: return reinterpret_cast<const void *>(&k_tile_queue<NMODE, VAR>);
    case kKernelRooted: return reinterpret_cast<const void *>(&k_tile_rooted<NMODE, VAR>);
    case kKernelResident:
      return reinterpret_cast<const void *>(&k_tile_resident<NMODE, VAR, kResidentThreads[0]>);
    case kKernelResident + 1:
      return reinterpret_cast<const void *>(&k_tile_resident<NMODE, VAR, kResidentThreads[1]>);
    default:
      return reinterpret_cast<const void *>(&k_tile_resident<NMODE, VAR, kResidentThreads[2]>);
  }
}

// var: 1 the integer subtractions (n = 1, 2), 2 the reference's Newton loop
// literally (a test of the fast paths).
template <int NMODE>
const void *kernel_of_n(int k, int var) {
  if (var == 2) return kernel_of_nv<NMODE, 2>(k);
  if (var == 1 && NMODE != kNGeneral) return kernel_of_nv<NMODE, 1>(k);
  return kernel_of_nv<NMODE, 0>(k);
}

const void *kernel_of(int k, int nmode, int var) {
  switch (nmode) {
    case kNOne: return kernel_of_n<kNOne>(k, var);
    case kNTwo: return kernel_of_n<kNTwo>(k, var);
    default: return kernel_of_n<kNGeneral>(k, var);
  }
}

int variant(const StepArgs &a) { return a.erode_generic ? 2 : a.erode_isub ? 1 : 0; }

}  // namespace

size_t tile_bytes(size_t total) {
  TileBufs b{};
  tile_carve(&b, nullptr, total);
  return reinterpret_cast<size_t>(b.queue) + (total * sizeof(int32_t) + 255) / 256 * 256;
}

void tile_carve(TileBufs *b, void *base, size_t total) {
  uintptr_t p = reinterpret_cast<uintptr_t>(base);
  auto take = [&](size_t bytes) -> uintptr_t {
    const uintptr_t at = p;
    p += (bytes + 255) / 256 * 256;
    return at;
  };
  b->code = reinterpret_cast<uint8_t *>(take(total * kWalkCells));
  b->planes = reinterpret_cast<uint32_t *>(take(total * 256 * sizeof(uint32_t)));
  b->local = reinterpret_cast<uint16_t *>(take(total * kWalkCells * sizeof(uint16_t)));
  b->inflow = reinterpret_cast<uint32_t *>(take(total * kSlots * sizeof(uint32_t)));
  b->sink = reinterpret_cast<unsigned long long *>(take(total * 2 * kSlots * sizeof(unsigned long long)));
  b->link = reinterpret_cast<uint32_t *>(take(total * kSlots * sizeof(uint32_t)));
  b->start = reinterpret_cast<uint32_t *>(take(total * kSlots * sizeof(uint32_t)));
  b->nstart = reinterpret_cast<int32_t *>(take(total * sizeof(int32_t)));
  b->done = reinterpret_cast<unsigned long long *>(take(total * kWalkH * sizeof(unsigned long long)));
  b->state = reinterpret_cast<int32_t *>(take(total * sizeof(int32_t)));
  b->queue = reinterpret_cast<int32_t *>(take(total * sizeof(int32_t)));
}

int append_walk_tiles(int r, int W, int H, Tile *out, int cap) {
  if (W <= 4 || H <= 4) return 0;  // no cell has a receiver or rises
  const int ntx = (W + kWalkW - 1) / kWalkW, nty = (H + kWalkH - 1) / kWalkH;
  if ((long long)ntx * nty > cap) return -1;
  int n = 0;
  for (int y = 0; y < nty; y++)
    for (int x = 0; x < ntx; x++) out[n++] = Tile{r, x * kWalkW, y * kWalkH, ntx};
  return n;
}

cudaError_t launch_tile_drain(const StepArgs &a, cudaStream_t s) {
  if (a.tb.n == 0) return cudaSuccess;
  k_tile_drain<<<a.tb.n, kDrainThreads, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_tile_links(const StepArgs &a, cudaStream_t s) {
  if (a.tb.n == 0) return cudaSuccess;
  k_tile_links<<<(a.tb.n + 7) / 8, 256, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_tile_counts(const StepArgs &a, cudaStream_t s) {
  if (a.tb.n == 0) return cudaSuccess;
  k_tile_counts<<<a.tb.n, kWalkThreads, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_tile_erode(const StepArgs &a, const TileRoom &room, cudaStream_t s) {
  StepArgs args = a;
  void *params[] = {&args};
  const int var = variant(a);
  // Resident tiles wait for one another: a cooperative launch, of the widest
  // blocks that all fit. 768 threads for one tile an SM measured the same as
  // 384.
  for (int w = kResidentWidths - 1; w >= 0; w--)
    if (a.tb.n <= room.resident[w])
      return cudaLaunchCooperativeKernel(kernel_of(kKernelResident + w, a.nmode, var), dim3(a.tb.n),
                                         dim3(kResidentThreads[w]), params, sizeof(TileSmem), s);
  return cudaLaunchKernel(kernel_of(kKernelRooted, a.nmode, var), dim3(a.tb.n), dim3(kRootedThreads),
                          params, sizeof(RootedSmem), s);
}

cudaError_t launch_tile_rest(const StepArgs &a, const TileRoom &room, cudaStream_t s) {
  if (a.tb.n <= room.resident[0]) return cudaSuccess;
  StepArgs args = a;
  void *params[] = {&args};
  const int var = variant(a);
  if (a.nmode == kNOne) {
    cudaError_t e = cudaLaunchKernel(kernel_of(kKernelPull, a.nmode, var), dim3(a.tb.n),
                                     dim3(kPullThreads), params, 0, s);
    if (e != cudaSuccess) return e;
    k_tile_mark<<<(a.tb.n + 7) / 8, 256, 0, s>>>(a);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  if (a.nmode != kNOne || a.tb.n >= kFrontCells / kWalkCells) {  // its blocks wait for one another
    const cudaError_t e =
        cudaLaunchCooperativeKernel(kernel_of(kKernelFront, a.nmode, var), dim3(room.front),
                                    dim3(kFrontThreads), params, 0, s);
    if (e != cudaSuccess) return e;
  }
  const int n = a.tb.n < room.queued ? a.tb.n : room.queued;
  return cudaLaunchKernel(kernel_of(kKernelQueue, a.nmode, var), dim3(n), dim3(kWalkThreads), params,
                          sizeof(TileSmem), s);
}

cudaError_t prepare_tile_kernels(int nmode, int sms, int tiles, TileRoom *room) {
  // blocks of kernel k on the GPU at once, whichever its arithmetic
  auto fit = [&](int k, int threads, size_t bytes, int *blocks) -> cudaError_t {
    int least = 1 << 20;
    for (int var = 0; var < 3; var++) {
      const void *f = kernel_of(k, nmode, var);
      cudaError_t e = cudaSuccess;
      if (bytes) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
      if (e != cudaSuccess) return e;
      int occ = 0;
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, f, threads, bytes);
      if (e != cudaSuccess) return e;
      least = occ < least ? occ : least;
    }
    *blocks = least * sms;
    return *blocks > 0 ? cudaSuccess : cudaErrorLaunchOutOfResources;
  };
  for (int w = kResidentWidths - 1; w >= 0; w--) {
    const cudaError_t e =
        fit(kKernelResident + w, kResidentThreads[w], sizeof(TileSmem), &room->resident[w]);
    if (e != cudaSuccess) return e;
    if (tiles <= room->resident[w]) {  // no launch needs narrower blocks, or the kernels below
      for (int v = 0; v < w; v++) room->resident[v] = room->resident[w];
      return cudaSuccess;
    }
  }
  int any = 0;
  cudaError_t e = fit(kKernelRooted, kRootedThreads, sizeof(RootedSmem), &any);
  if (e == cudaSuccess && (nmode != kNOne || tiles >= kFrontCells / kWalkCells))
    e = fit(kKernelFront, kFrontThreads, 0, &room->front);
  if (e == cudaSuccess) e = fit(kKernelQueue, kWalkThreads, sizeof(TileSmem), &room->queued);
  return e;
}

}  // namespace fs
