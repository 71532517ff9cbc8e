// fs_noalloc.cu -- fs_step_noalloc: FastScape timesteps on a caller-owned
// device elevation buffer, with every piece of scratch memory in one static
// device array, so the call itself never allocates.
//
// Who needs this: callers that are not allowed to allocate device memory
// once they are running -- a host application that hands the library a
// device pointer from its own memory pool and forbids outside cudaMalloc
// (allocating would bypass its accounting or fragment its arena), code that
// runs on a latency-critical path where a cudaMalloc/cudaFree would
// synchronize the device, and plugins that must keep a fixed memory
// footprint decided at load time. fs_create allocates per model; this entry
// point allocates nothing.
//
// Limits and sharing:
//   * grids of at most FS_NOALLOC_MAX_CELLS cells (width*height); larger
//     grids are rejected with FS_ERR_ARG;
//   * the scratch array (~41 MB: receivers, drainage counts, the tile walk's
//     arrays for the most tiles a grid within the limit can have -- a
//     5-cell-wide one, 1639 -- the erosion table for every possible count,
//     stencil tiles, descriptors and the control block) lives in the library
//     image, so every GPU that loads the library holds it until the process
//     exits;
//   * every call on a device uses the same array and it keeps the last
//     call's contents; calls that overlap on the GPU race on it. The library
//     serializes its own calls (a host mutex, and each call waits for its
//     stream before returning), so two calls of this entry point do not
//     overlap; what the caller must still order against the call's stream is
//     its own work on d_h (kernels or copies in flight on other streams);
//   * the input is checked for NaN/Inf first, as fs_set_elevation does
//     (FS_ERR_NONFINITE, d_h untouched);
//   * the first call on a device looks up the array's device address
//     (cudaGetSymbolAddress) and the walk kernel's occupancy; make that first
//     call before any stream capture. Later calls look the address up again
//     and start over when it moved (after a cudaDeviceReset the module is
//     loaded afresh and the array comes back zeroed).
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>

#include "fastscape_gb300.h"
#include "fs_internal.h"

namespace {

constexpr size_t kMaxCells = FS_NOALLOC_MAX_CELLS;
constexpr size_t kTabRecords = kMaxCells + 1;  // counts 0..kMaxCells
constexpr int kMaxTiles = 4096;                // receiver tiles
constexpr size_t kMaxWalkTiles = kMaxCells / 5 / fs::kWalkH + 1;  // 5 cells wide
constexpr int kMaxDevices = 64;

constexpr size_t align256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }

// Regions of the scratch array, each 256-byte aligned.
constexpr size_t kOffCtl = 0;
constexpr size_t kOffDesc = align256(kOffCtl + sizeof(fs::Ctl));
constexpr size_t kOffRtiles = align256(kOffDesc + sizeof(fs::RealDesc));
constexpr size_t kOffWtiles = align256(kOffRtiles + kMaxTiles * sizeof(fs::Tile));
constexpr size_t kOffTab = align256(kOffWtiles + kMaxWalkTiles * sizeof(fs::Tile));
constexpr size_t kOffAmb = align256(kOffTab + kTabRecords * fs::kTabStride * sizeof(double));
constexpr size_t kOffAmbR = align256(kOffAmb + kMaxCells * sizeof(int32_t));
constexpr size_t kOffCount = align256(kOffAmbR + kMaxCells * sizeof(int32_t));
constexpr size_t kOffRec = align256(kOffCount + kMaxCells * sizeof(uint32_t));
constexpr size_t kOffTiles = align256(kOffRec + kMaxCells);
constexpr size_t kTileScratch = align256(kMaxWalkTiles * fs::kWalkTileBytes + 16 * 256);
constexpr size_t kScratchBytes = kOffTiles + kTileScratch;

// The scratch. Host code must not use this name as a device address (on the
// host it is only a stand-in); the address comes from cudaGetSymbolAddress.
static __device__ __align__(256) unsigned char g_scratch[kScratchBytes];

// Host copies for the parameters last uploaded: erosion table, tiles.
static double g_host_tab[kTabRecords * fs::kTabStride];
static fs::Tile g_host_tiles[2][kMaxTiles];  // receiver and walk tiles

struct DeviceState {
  bool ready = false;
  unsigned char *base = nullptr;  // device address of g_scratch
  fs::TileRoom room[3];          // per n mode
  bool tab_valid = false;
  fs_params tab_params{};
};

DeviceState g_dev[kMaxDevices];
std::mutex g_mutex;

int fail(int status, const char *msg) {
  char buf[256];
  std::snprintf(buf, sizeof(buf), "fs_step_noalloc: %s", msg);
  return fs::record_error(status, buf);
}

int cuda_fail(cudaError_t e, const char *what) {
  char buf[200];
  std::snprintf(buf, sizeof(buf), "%s: %s", what, cudaGetErrorString(e));
  return fail(FS_ERR_CUDA, buf);
}

bool same_params(const fs_params &a, const fs_params &b) {
  return std::memcmp(&a, &b, sizeof(fs_params)) == 0;
}

int setup_device(int dev, DeviceState &d) {
  void *ptr = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&ptr, g_scratch);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(scratch)");
  if (d.ready && d.base == ptr) return FS_OK;
  // first call on this device, or the module was reloaded (the array is
  // zeroed and may sit elsewhere): nothing cached about it holds any more
  d = DeviceState{};
  if (fs::tile_bytes(kMaxWalkTiles) > kTileScratch) return fail(FS_ERR_CUDA, "scratch too small");
  int sms = 0;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaDeviceGetAttribute");
  for (int nm = 0; nm < 3; nm++) {
    e = fs::prepare_tile_kernels(nm, sms, static_cast<int>(kMaxWalkTiles), &d.room[nm]);
    if (e != cudaSuccess) return cuda_fail(e, "tile kernels");
  }
  d.base = static_cast<unsigned char *>(ptr);
  d.ready = true;
  return FS_OK;
}

}  // namespace

extern "C" int fs_step_noalloc(double *d_h, int width, int height, const fs_params *params,
                               int nsteps, void *stream) {
  if (!d_h || !params) return fail(FS_ERR_ARG, "d_h and params must not be NULL");
  if (width < 3 || height < 3) return fail(FS_ERR_ARG, "width and height must be >= 3");
  if (static_cast<long long>(width) * height > static_cast<long long>(kMaxCells)) {
    char buf[160];
    std::snprintf(buf, sizeof(buf),
                  "grid of %lld cells exceeds the static scratch limit of %lld cells "
                  "(FS_NOALLOC_MAX_CELLS); use fs_create for larger grids",
                  static_cast<long long>(width) * height, static_cast<long long>(kMaxCells));
    return fail(FS_ERR_ARG, buf);
  }
  if (nsteps < 0) return fail(FS_ERR_ARG, "nsteps must be >= 0");
  const fs_params &p = *params;
  if (!(p.dr_orth > 0) || !(p.dr_diag > 0) || !(p.cell_area > 0) || !(p.tol >= 0) ||
      !std::isfinite(p.keq) || !std::isfinite(p.neq) || !std::isfinite(p.meq) ||
      !std::isfinite(p.ueq) || !std::isfinite(p.dt))
    return fail(FS_ERR_ARG, "parameters must be finite, dr and cell_area > 0, tol >= 0");
  fs::Tile *rt = g_host_tiles[0], *wt = g_host_tiles[1];

  std::lock_guard<std::mutex> lock(g_mutex);
  const int nrt = fs::append_tiles(fs::receiver_rows(1, &width, &height), 0, width, height, rt, kMaxTiles);
  const int nwt = fs::append_walk_tiles(0, width, height, wt, kMaxWalkTiles);
  if (nrt < 0 || nwt < 0) return fail(FS_ERR_ARG, "grid too elongated for the static tile list");
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  if (dev < 0 || dev >= kMaxDevices) return fail(FS_ERR_ARG, "device index out of range");
  DeviceState &d = g_dev[dev];
  if (int st = setup_device(dev, d)) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);

  fs::Ctl *ctl = reinterpret_cast<fs::Ctl *>(d.base + kOffCtl);
  fs::RealDesc *desc = reinterpret_cast<fs::RealDesc *>(d.base + kOffDesc);
  fs::Tile *d_rt = reinterpret_cast<fs::Tile *>(d.base + kOffRtiles);
  fs::Tile *d_wt = reinterpret_cast<fs::Tile *>(d.base + kOffWtiles);
  double *tab = reinterpret_cast<double *>(d.base + kOffTab);

  if (!d.tab_valid || !same_params(d.tab_params, p)) {
    fs::fill_table_range(p.keq, p.neq, p.meq, p.dt, p.dr_orth, p.dr_diag, p.cell_area, 0,
                         static_cast<long long>(kTabRecords), g_host_tab);
    e = cudaMemcpyAsync(tab, g_host_tab, sizeof(g_host_tab), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
      d.tab_valid = false;
      return cuda_fail(e, "upload(erosion table)");
    }
    d.tab_params = p;
    d.tab_valid = true;
  }

  const int size = width * height;
  fs::RealDesc rd{};
  rd.W = width;
  rd.H = height;
  rd.size = size;
  rd.off = 0;
  rd.lvl_base = 0;
  rd.nring = fs::ring_cells(width, height);
  rd.u_dt = p.ueq * p.dt;
  rd.tol = fs::make_tolerance(p.tol);
  rd.g_orth = static_cast<float>(1.0 / p.dr_orth);
  rd.g_diag = static_cast<float>(1.0 / p.dr_diag);
  rd.gmax = rd.g_orth > rd.g_diag ? rd.g_orth : rd.g_diag;
  rd.dr_orth = p.dr_orth;
  rd.dr_diag = p.dr_diag;
  rd.rdr_orth_n = fs::neg_recip_dr(p.dr_orth);
  rd.rdr_diag_n = fs::neg_recip_dr(p.dr_diag);
  rd.tab = tab;
  rd.tab_cap = static_cast<int>(kTabRecords);

  fs::StepArgs a{};
  a.h = d_h;
  a.rec = reinterpret_cast<int8_t *>(d.base + kOffRec);
  a.amb = reinterpret_cast<int32_t *>(d.base + kOffAmb);
  a.amb_r = reinterpret_cast<int32_t *>(d.base + kOffAmbR);
  a.desc = desc;
  a.ctl = ctl;
  a.nreal = 1;
  a.rtiles = d_rt;
  a.nrtiles = nrt;
  a.rrows = fs::receiver_rows(1, &width, &height);
  fs::tile_carve(&a.tb, d.base + kOffTiles, nwt);
  a.tb.tiles = d_wt;
  a.tb.n = nwt;
  a.tb.desc = desc;
  a.tb.count = reinterpret_cast<uint32_t *>(d.base + kOffCount);
  a.nmode = (p.neq == 1.0) ? fs::kNOne : (p.neq == 2.0) ? fs::kNTwo : fs::kNGeneral;
  a.neq = p.neq;
  a.do_erode = 1;
  a.timeout_ns = 2000000000ull;

  // Start state: descriptors and tiles of this grid, control words zeroed,
  // rings without receivers.
  e = cudaMemcpyAsync(desc, &rd, sizeof(rd), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess && nrt > 0)
    e = cudaMemcpyAsync(d_rt, rt, nrt * sizeof(fs::Tile), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(d_wt, wt, nwt * sizeof(fs::Tile), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(ctl, 0, sizeof(fs::Ctl), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(a.rec, 0xff, size, s);
  // NaN/Inf in the caller's field is refused before any timestep, like
  // fs_set_elevation refuses it
  if (e == cudaSuccess) e = fs::launch_check_finite(d_h, size, ctl, s);
  int in_err = 0;
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(&in_err, &ctl->err, sizeof(int), cudaMemcpyDeviceToHost, s);
  // the host copies above read static buffers this call rewrites next time
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_fail(e, "scratch reset");
  if (in_err == FS_ERR_NONFINITE) return fail(FS_ERR_NONFINITE, "input holds NaN or Inf");
  if (in_err != 0) return fail(in_err, "input check failed on the device");
  if (nwt == 0) return FS_OK;  // no interior: a timestep changes nothing

  for (int i = 0; i < nsteps; i++) {
    e = fs::launch_receivers_fast(a, s);
    if (e == cudaSuccess) e = fs::launch_tile_drain(a, s);
    if (e == cudaSuccess) e = fs::launch_tile_links(a, s);
    if (e == cudaSuccess) e = fs::launch_tile_erode(a, d.room[a.nmode], s);
    if (e == cudaSuccess) e = fs::launch_tile_rest(a, d.room[a.nmode], s);
    if (e != cudaSuccess) return cuda_fail(e, "timestep launch");
  }
  fs::Ctl h_ctl;
  e = cudaMemcpyAsync(&h_ctl, ctl, sizeof(fs::Ctl), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_fail(e, "status read-back");
  if (h_ctl.err != 0) return fail(h_ctl.err, "a timestep failed on the device");
  if (h_ctl.steps_done != nsteps) return fail(FS_ERR_CUDA, "not every timestep completed");
  return FS_OK;
}
