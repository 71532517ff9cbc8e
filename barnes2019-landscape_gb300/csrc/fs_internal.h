// fs_internal.h -- shared between the host side (fs_model.cu, fs_noalloc.cu)
// and the kernels (fs_kernels.cu). Not part of the public ABI.
//
// Every timestep runs over a batch of realizations (a single model is a
// batch of one). Realization r owns the cells [off_r, off_r + size_r) of
// every per-cell and per-position array and the level-table entries
// [lvl_base_r, lvl_base_r + size_r + 2); cell indices stored in `ent` are
// local to the realization (c = y*W_r + x).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

namespace fs {

// Batch-wide control block, zeroed (but for `queued`) before every call. `err` holds the first
// error status of the current call; the words from `amb` on start every
// timestep at zero (k_tile_drain: a memset node took 2.5 us of a 55 us step).
struct Ctl {
  int err;                 // FS_OK or first FS_ERR_* seen by any kernel
  int err_detail;          // phase code where err was raised
  int abort_k;             // > 0: a drainage count >= its realization's table
                           // capacity was met; the timestep stopped before
                           // touching h
  int steps_done;          // timesteps completed in the current fs_step call
  int abort_r;             // realization (of the batch) that raised abort_k
  int pad0[3];
  // --- zero when a timestep starts ---
  int amb;                 // cells queued by the receiver filter
  int left;                // cells still to erode in trees that leave their
                           // tile (k_tile_queue), or tiles finished (resident)
  unsigned int qtail, qhead;  // pushes to and pops from the tile queue
  int progress;            // moves, like left, while tiles get further (tiles_moved)
  unsigned int bar;        // blocks' arrivals (k_tile_front, k_test_wait)
  unsigned int front[3];   // k_tile_front: cells of a round (rotating)
  // --- kept ---
  int queued;              // cells that the last receiver filter queued
};
constexpr size_t kCtlCallResetBytes = offsetof(Ctl, queued);
constexpr size_t kCtlResetOffset = offsetof(Ctl, amb);
constexpr size_t kCtlResetBytes = kCtlCallResetBytes - kCtlResetOffset;

// Per-realization counters, reset before every ordering.
struct RealCtl {
  int top;                 // pits appended to level 0 (after the rings)
  int nlevels;             // levels found (k_cta_order_accum, k_net_follow)
};

// The Newton tolerance in the forms the erosion compares with.
struct Tolerance {
  double tol;
  long long bits;          // of tol (magnitude compares as integers)
  float lo_f;              // an FP32 value <= tol*(1-2^-20)
  uint32_t q_hi, y_hi;     // upper words at most tol*(1-2^-8)'s and
                           // tol*2^39's (steps surely below tol)
  uint32_t above_hi;       // and tol*(1+2^-7)'s (steps surely above)
};

// Read-only description of one realization.
struct RealDesc {
  int W, H, size;
  int off;                 // first cell / position of the realization
  int lvl_base;            // first entry of its level table
  int nring;               // ring cells, pre-placed at ent[off, off+nring)
  double u_dt;             // ueq*dt
  Tolerance tol;
  float g_orth, g_diag, gmax;  // FP32 1/dr for the receiver filter
  double dr_orth, dr_diag;
  double rdr_orth_n, rdr_diag_n;  // -RN(1/dr) for the tabled receiver
                                  // slope division; 0: divide in IEEE FP64
  const double *tab;       // erosion table, kTabStride doubles per count
  int tab_cap;             // counts k < tab_cap are in the table
  int tile0;               // first of its walk tiles
  int id;                  // its number in the batch
};

// A 2-D tile of one realization for the stencil kernels.
struct Tile {
  int r;                   // realization
  int x0, y0;              // grid coordinates of the tile's first cell
  int ntx;                 // walk tiles: tiles per row of the realization
};

// Receiver code of an interior cell without a lower neighbour. The ABI
// reports it as FS_NO_FLOW (-1), like the rings; internally it marks the
// level-0 cells that are uplifted (fastscape_RB.cpp:291-295).
constexpr int kPit = -2;

// Erosion table: one 64-byte record per drainage count k (cells), holding
// for each direction class (0 orthogonal, 1 diagonal) at doubles 4*cls+0..3:
//   F = keq*dt*pow(k*cell_area, meq)/pow(dr_cls, neq)  (fastscape_RB.cpp:315)
//   D = 1 + F          (the n = 1 Newton denominator, fastscape_RB.cpp:322)
//   R = RN(1/D)        (reciprocal for the correctly rounded division)
//   -R                 (the same, negated)
constexpr int kTabStride = 8;

// Tiles: receivers over the interior [2, W-3]^2; donors over [1, W-2]^2
// with tiles starting at x = 0, 128, 256, ... (four cells per thread, so a
// row of a realization whose byte offset is a multiple of 4 is stored in
// whole words). Tall tiles (a thread slides down 12 rows of receivers, 8 of
// donors) spread each block's fixed costs -- staging halo, tile-wide bound,
// queue scan and atomic -- over more cells; measured fastest from 1000^2 up
// and within microseconds below.
constexpr int kRxTile = 32, kRyTile = 96, kRySmall = 32;
constexpr int kDxTile = 128, kDyTile = 64;

// The donor kernel reads rec as aligned 32-bit words around each tile row,
// up to 8 bytes before the first and 144 bytes past the last byte of a
// realization: rec buffers keep kRecPad readable bytes on both sides that no
// kernel writes while the donor kernel runs.
constexpr size_t kRecPad = 256;

// Where an error was detected (Ctl::err_detail).
enum ErrPhase : int {
  kPhaseNone = 0,
  kPhaseBarrier = 1,
  kPhaseOrder = 2,
  kPhaseErode = 3,
  kPhaseTest = 4,
};

// How pow(x, n) and pow(x, n-1) are evaluated inside the Newton loop.
enum NMode : int {
  kNGeneral = 0,  // CUDA pow (not bit-identical to glibc)
  kNOne = 1,      // pow(x,1) = x, pow(x,0) = 1: exact
  kNTwo = 2,      // pow(x,2) = x*x, pow(x,1) = x
};

// Walk tiles: the grid cut into rectangles of 64 x 32 cells from its first
// cell on (fs_tile.cu). Every realization owns ntx*nty of them, row by row;
// tile t's cells are numbered c = 64*y + x inside it. Cells on a tile's edge
// that trade water with other tiles are named by their perimeter slot: 0..63
// the top row, 64..127 the bottom row, 128..159 the left and 160..191 the
// right column (corners belong to the rows). A tile's sinks are its cells
// through which water of other tiles leaves it: slot s for the exit cell at
// slot s, 192 + s for the cell above a root that the water entering at slot s
// (and at other slots) ends in.
constexpr int kWalkW = 64, kWalkH = 32;
constexpr int kWalkCells = kWalkW * kWalkH;
constexpr int kSlots = 2 * kWalkW + 2 * kWalkH;
// Cell codes inside a tile: 0..7 the direction of a receiver inside the
// tile, kCodeExit | direction of one outside, kCodeRoot no receiver,
// kCodeOutside past the grid's edge.
constexpr int kCodeRoot = 8, kCodeOutside = 9, kCodeExit = 16;

struct TileBufs {
  const Tile *tiles;       // every walk tile of the batch
  const int32_t *list;     // the tiles of this launch (null: all, in order)
  int n;                   // how many
  const RealDesc *desc;    // every realization (not only the active ones)
  uint8_t *code;           // [t][2048] cell codes
  uint32_t *planes;        // [t][4][64] bit planes of the directions' three
                           // bits and of "has a receiver", 32 cells a word
  uint16_t *local;         // [t][2048] cells drained inside the tile
  uint32_t *inflow;        // [t][192] cells drained from other tiles, by slot
  unsigned long long *sink;  // [t][384] cells << 16 | edges still to come in
  uint32_t *link;          // [t][192] slot -> sink, and that exit's target
  uint32_t *start;         // [t][192] exits that wait for nothing
  int32_t *nstart;         // [t] how many
  unsigned long long *done;  // [t][32] rows of cells whose elevation is final
  int32_t *state;          // [t] kTileQueued | kTileAgain
  int32_t *queue;          // [n] ring of queued tiles + 1, 0 where empty
  uint32_t *count;         // drainage count per cell (grid layout)
};
// Bytes of one tile in the arrays above (12 KB), before rounding.
constexpr size_t kWalkTileBytes = kWalkCells * (1 + 2) + 256 * 4 + kSlots * (4 + 16 + 4 + 4) +
                                  kWalkH * 8 + 4 + 4 + 4;
// Bytes of the per-tile arrays, and their pointers inside one allocation of
// tile_bytes(total) bytes (256-byte aligned).
size_t tile_bytes(size_t total);
void tile_carve(TileBufs *b, void *base, size_t total);
// Walk tiles of realization r appended to out (capacity cap), as
// append_tiles: none where nothing flows, in grids without an interior (whose
// tiles, three cells wide, would take 128 bytes a cell).
int append_walk_tiles(int r, int W, int H, Tile *out, int cap);

// Arrays indexed by position i in the level order (the reference's stack):
//   ent[i]   cell index (local); level 0 starts with the two rings (fixed)
//            followed by the pits of this timestep; each level lists the
//            donors of the level before it, a receiver's donors contiguous
//   pdir[i]  receiver direction of ent[i] (0..7)
//   acc[i]   drainage cell count of ent[i]
//   par[i]   position of ent[i]'s receiver (levels >= 1)
struct StepArgs {
  double *h;
  int8_t *rec;
  uint8_t *mask;
  int32_t *ent;
  uint8_t *pdir;
  uint32_t *acc;
  int32_t *par;
  int32_t *amb;            // queued cells (global index) of the filter
  int32_t *amb_r;          // and their realization
  int32_t *lvl_off;        // per realization: size+2 local level offsets
  const RealDesc *desc;
  RealCtl *rctl;
  Ctl *ctl;
  int nreal;
  const Tile *rtiles;
  int nrtiles, rrows;      // receiver tiles, and their rows (receiver_rows)
  const Tile *dtiles;
  int ndtiles;
  int nmode;
  double neq;
  int do_erode;            // 0: ordering + accumulation only
  int erode_isub;          // 1: the n = 1 / n = 2 erosion subtracts
                           // elevations in integer arithmetic (host-side
                           // launch choice)
  int erode_generic;       // 1: the reference's Newton loop literally, for
                           // every n (a test of the fast paths)
  unsigned long long timeout_ns;
  TileBufs tb;
};

// Largest batch one walk launch handles.
constexpr int kMaxReal = 4096;
// Kernel launchers (fs_kernels.cu). All are asynchronous on `s`.
cudaError_t launch_receivers_exact(const StepArgs &a, cudaStream_t s);
// hmap: a single grid's elevation as a {W, H} map of 64-bit elements with
// {36, rows + 2} boxes (make_receiver_map): the filter stages its tiles by TMA.
cudaError_t launch_receivers_fast(const StepArgs &a, cudaStream_t s,
                                  const CUtensorMap *hmap = nullptr);
bool make_receiver_map(CUtensorMap *m, const double *h, int W, int H, int rows);
cudaError_t launch_donors_level0(const StepArgs &a, cudaStream_t s);
// The tile walk (fs_tile.cu): drainage inside the tiles, drainage between
// them, and the counts alone or the erosion. `resident`, `queued` and `front`
// are the blocks that k_tile_resident, k_tile_queue and k_tile_front can
// keep on the GPU at once.
constexpr int kResidentWidths = 3;  // of k_tile_resident's blocks, narrowest first
struct TileRoom {
  int resident[kResidentWidths] = {}, queued = 0, front = 0;
};
cudaError_t launch_tile_drain(const StepArgs &a, cudaStream_t s);
cudaError_t launch_tile_links(const StepArgs &a, cudaStream_t s);
cudaError_t launch_tile_counts(const StepArgs &a, cudaStream_t s);
cudaError_t launch_tile_erode(const StepArgs &a, const TileRoom &room, cudaStream_t s);
cudaError_t launch_tile_rest(const StepArgs &a, const TileRoom &room, cudaStream_t s);
// Raises the shared-memory limits of the kernels that launches of up to `tiles`
// tiles take, and counts the room for the n mode on a GPU of sms SMs (a few
// microseconds a kernel: 1000^2 is created in 1.63 instead of 1.71 ms without
// those it never takes).
cudaError_t prepare_tile_kernels(int nmode, int sms, int tiles, TileRoom *room);
// The per-realization walk (batches of many small realizations): one CTA per
// realization orders and accumulates, then uplifts and erodes (skipped on an
// abort or error).
cudaError_t launch_cta_order(const StepArgs &a, int sms, cudaStream_t s);
cudaError_t launch_cta_erode(const StepArgs &a, int sms, cudaStream_t s);
cudaError_t launch_check_finite(const double *h, long long n, Ctl *ctl, cudaStream_t s);
cudaError_t launch_philox_field(double *h, int W, int H, uint64_t seed, cudaStream_t s);
cudaError_t launch_place_rings(int32_t *ent, int W, int H, cudaStream_t s);
// Codes and counts of a grid without receivers: -1 on the rings, kPit inside;
// every cell drains itself.
cudaError_t launch_no_receivers(int8_t *rec, uint32_t *count, int W, int H, cudaStream_t s);
cudaError_t launch_test_wait(Ctl *ctl, int blocks, unsigned long long timeout_ns,
                             cudaStream_t s);

// The drainage network of one realization (fs_network.cu), for read-backs.
struct NetArgs {
  const int8_t *rec;
  const uint32_t *count;      // drainage counts (not for the levels)
  int n, W;                   // cells, row length
  unsigned long long *words;  // [n] scratch
};
// Levels into out[n]; rctl->nlevels becomes the number of levels.
cudaError_t launch_net_levels(const NetArgs &a, RealCtl *rctl, Ctl *ctl, int32_t *out,
                              cudaStream_t s);
// First position of each tree of the depth-first order into starts, the
// number of trees into sums[net_sums(n)].y, and the words that
// launch_net_order turns into the order (which may take starts' place).
int net_sums(int n);
cudaError_t launch_net_trees(const NetArgs &a, int2 *sums, int32_t *starts, cudaStream_t s);
cudaError_t launch_net_order(const NetArgs &a, Ctl *ctl, int32_t *out, cudaStream_t s);
cudaError_t launch_net_receivers(const NetArgs &a, int32_t *out, cudaStream_t s);
cudaError_t launch_net_receiver_index(const NetArgs &a, long long *out, cudaStream_t s);
cudaError_t launch_net_area(const NetArgs &a, double cell_area, double *out, cudaStream_t s);

// Host helpers shared by the entry points.
Tolerance make_tolerance(double tol);
// -RN(1/dr) when the tabled division covers dr (1 <= dr <= 2^60), else 0.
double neg_recip_dr(double dr);
int ring_cells(int W, int H);
// Rows of the receiver tiles of n realizations: 96, or 32 where 96 would give
// the 152 SMs less than a block each (receivers of 100^2 21.6 -> 18.7 us, of
// 512^2 22.6 -> 20.5; 1000^2, of 352 tiles, 25.9 at 96 rows and 27.6 at 32,
// whose halo costs 6% instead of 2%).
int receiver_rows(int n, const int *W, const int *H);
// Appends the receiver (rows > 0) or donor (rows = 0) tiles of realization r to
// out (capacity cap); returns the number appended, or -1 if out is full.
int append_tiles(int rows, int r, int W, int H, Tile *out, int cap);
// Erosion-table records for counts [k0, k1) into rec (kTabStride doubles
// each), single-threaded.
void fill_table_range(double keq, double neq, double meq, double dt, double dr_orth,
                      double dr_diag, double cell_area, long long k0, long long k1,
                      double *rec);

// Stores `msg` as this thread's fs_last_error() text; returns status.
int record_error(int status, const char *msg);

}  // namespace fs
