// noalloc.cu — a 2D solve that allocates nothing.
//
// Some callers cannot allocate device memory at the moment they need a cut:
// real-time frame loops that must not stall on the allocator (a cudaMalloc
// can synchronise the device and take milliseconds), and hosts that hand this
// library a fixed memory budget up front and forbid allocations after it.
// jfc_solve_grid2d_noalloc serves them: the whole working set of the solve
// (residual graph, heights, labels, tile tables, work queues, counters) lives
// in one file-scope device array of fixed size, so the call itself performs no
// cudaMalloc / cudaFree / cudaMallocHost and uses no allocating library
// routine.  The caller passes device inputs and outputs.  The call reads a few
// counters back between relabel cycles, so it synchronises `stream` before it
// returns.
//
// Limits and sharing:
//  * grids whose padded size (width rounded up to 32, height rounded up to
//    16) is at most kMaxNodes = 524,288 nodes — e.g. 1024 x 512 or the
//    600 x 450 / 640 x 480 images that ship with the reference; larger grids
//    are rejected with JFC_ERR_INVALID_ARG;
//  * the array (about 13.5 MB) is held by every GPU that loads the library,
//    until the process exits;
//  * every call shares the array and it keeps the last call's contents (the
//    solve clears what must start at zero); calls that overlap on the GPU —
//    on two streams, or from two threads — race and corrupt each other;
//  * the first call on a device looks up the array's device address
//    (cudaGetSymbolAddress, once per device, with that device current); make
//    that first call before any stream capture begins;
//  * the caller's current device is restored before the call returns.
#include <algorithm>
#include <cstring>
#include <mutex>

#include "engine.h"

namespace {

constexpr int kMaxNodes = 1 << 19;                 // padded nodes
constexpr int kMaxTiles = kMaxNodes / (32 * 8);    // tiles at the smallest tile height
constexpr size_t al(size_t v) { return (v + 255) / 256 * 256; }
constexpr size_t kPlane = al(sizeof(int) * (size_t)kMaxNodes);
constexpr size_t kTileI = al(sizeof(int) * (size_t)kMaxTiles);
// layout of the scratch array
constexpr size_t kOffE = 0;
constexpr size_t kOffH = kOffE + kPlane;
constexpr size_t kOffR = kOffH + kPlane;            // 4 residual planes
constexpr size_t kOffLabel = kOffR + 4 * kPlane;
constexpr size_t kOffDesc = kOffLabel + al(kMaxNodes);
constexpr size_t kOffInfo = kOffDesc + al(sizeof(GridDev));
constexpr size_t kOffFlagPr = kOffInfo + al(sizeof(int4) * (size_t)kMaxTiles);
constexpr size_t kOffQPr = kOffFlagPr + kTileI;     // 4 queues
constexpr size_t kOffSum = kOffQPr + 4 * kTileI;
// the control block and, behind it, the grid's active tiles: read back together
constexpr size_t kOffCtr = kOffSum + 256;
constexpr size_t kOffGact = kOffCtr + sizeof(DevCounters);
// regions of the global relabel: the most a grid of kMaxNodes padded nodes has
// (kMaxNodes / 32 row words; one column of regions 1 word wide, or one row of
// regions 16 rows high)
constexpr int kMaxReg = kMaxNodes / (32 * 16) / JFC_WAVE_WORDS + kMaxNodes / 32 / JFC_WAVE_ROWS + 2;
constexpr size_t kOffDirty = kOffCtr + al(sizeof(DevCounters) + sizeof(int));
constexpr size_t kOffVf = kOffDirty + al(kMaxTiles);
constexpr size_t kOffReg = kOffVf + al(sizeof(uint4) * (size_t)(kMaxNodes / 32));
constexpr size_t kOffRrec = kOffReg + al(sizeof(int4) * (size_t)kMaxReg);
constexpr size_t kOffRflag = kOffRrec + al(sizeof(unsigned) * (size_t)kMaxReg);   // 2 flag arrays
constexpr size_t kOffBad = kOffRflag + 2 * al(kMaxReg);
constexpr size_t kBytes = kOffBad + 256;

std::mutex g_mu;
void* g_addr[128] = {nullptr};

// Restores the calling thread's current device when the call returns.
struct DeviceGuard {
  int prev = -1;
  DeviceGuard() { if (cudaGetDevice(&prev) != cudaSuccess) prev = -1; }
  ~DeviceGuard() { if (prev >= 0) cudaSetDevice(prev); }
};

// tile t of a single grid: {grid 0, tx, ty, tz 0}
__global__ void k_na_tile_info(int4* info, int tiles_x, int ntiles) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += gridDim.x * blockDim.x)
    info[t] = make_int4(0, t % tiles_x, t / tiles_x, 0);
}

// region k of a single grid of rx regions a row: {grid 0, x, y, first region 0}
__global__ void k_na_regions(int4* reg, int rx, int n) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
    reg[k] = make_int4(0, k % rx, k / rx, 0);
}

}  // namespace

// The working set of jfc_solve_grid2d_noalloc.  In host code this name is a
// host-side stand-in, not a device address: kernels get the address from
// cudaGetSymbolAddress (na_scratch below).
static __device__ __align__(256) unsigned char g_noalloc_scratch[kBytes];

namespace {

int na_scratch(int device, char** out) {
  std::lock_guard<std::mutex> lock(g_mu);
  if (device < 0 || device >= 128) return set_error(JFC_ERR_INVALID_ARG, "bad device index");
  if (!g_addr[device]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr) return cuda_status(e, "cudaGetSymbolAddress(no-allocation scratch)");
    g_addr[device] = p;
  }
  *out = (char*)g_addr[device];
  return JFC_OK;
}

cudaError_t na_copy(void* padded, const void* dense, size_t elem, int w, int h, int pitch, int Hp, bool to_dense,
                    cudaStream_t s) {
  cudaMemcpy3DParms p{};
  cudaPitchedPtr pad = make_cudaPitchedPtr(padded, (size_t)pitch * elem, (size_t)pitch, (size_t)Hp);
  cudaPitchedPtr den = make_cudaPitchedPtr(const_cast<void*>(dense), (size_t)w * elem, (size_t)w, (size_t)h);
  p.srcPtr = to_dense ? pad : den;
  p.dstPtr = to_dense ? den : pad;
  p.extent = make_cudaExtent((size_t)w * elem, (size_t)h, 1);
  p.kind = cudaMemcpyDeviceToDevice;
  return cudaMemcpy3DAsync(&p, s);
}

// Read back the control block into caller-stack memory (no pinned buffer).
int na_read(void* host, const void* dev, size_t bytes, cudaStream_t s) {
  JFC_CUDA(cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, s));
  JFC_CUDA(cudaStreamSynchronize(s));
  return JFC_OK;
}

// What a run of cycles reads back, with one wait.
struct NaRead {
  DevCounters ctr;
  int active;
};

int na_status(const NaRead& r) {
  if (r.ctr.error) return set_error(JFC_ERR_CUDA, "a device-side wait timed out in a persistent kernel (grid barrier, worklist or tile staging)");
  if (r.ctr.bfs_status == 2) return set_error(JFC_ERR_NOT_CONVERGED, "BFS pass budget exhausted");
  return JFC_OK;
}

// A run of up to kRun cycles { push-relabel phase, global relabel } and the exact
// relabel and the cut behind them, with one wait: what is not due returns at
// once (a loop on the device would need a graph, which allocates).  A launch
// that is not due costs 2.5 us, a wait 28: 15 grids of 7 to 20 cycles took 1.71
// to 2.95 ms with a wait per cycle, 1.49 to 2.65 in runs of 3, 1.47 to 2.57 in
// runs of 8, and the same in runs of 6 or 12.
constexpr int kRun = 8;
int na_run(TileSet& ts, const jfc_params& p, bool init, CycleState& cyc, cudaStream_t s, NaRead& r) {
  cyc.cycles = cyc.sweeps = cyc.passes = cyc.done = cyc.exact = 0;
  cyc.go = !init;
  cyc.max_cycles = init ? kRun + 1 : kRun;
  JFC_CUDA(cudaMemcpyAsync(&ts.d_ctr->cyc, &cyc, sizeof(cyc), cudaMemcpyHostToDevice, s));
  TileSet part = ts;
  if (init) {
    part.cyc_mode = 1;
    JFC_CUDA(launch_bfs(part, false, p.max_bfs_passes, s));
  }
  part.cyc_mode = 2;
  for (int k = 0; k < kRun; ++k) {
    JFC_CUDA(launch_pr_phase(part, 0, 0, s));
    JFC_CUDA(launch_bfs(part, false, p.max_bfs_passes, s));
  }
  part.cyc_mode = 3;
  JFC_CUDA(launch_bfs(part, false, p.max_bfs_passes, s));
  part.cyc_mode = 4;
  JFC_CUDA(launch_bfs(part, true, p.max_bfs_passes, s));
  static_assert(sizeof(DevCounters) % alignof(int) == 0 && sizeof(NaRead) >= sizeof(DevCounters) + sizeof(int), "");
  const int rc = na_read(&r, ts.d_ctr, offsetof(NaRead, active) + sizeof(int), s);
  cyc = r.ctr.cyc;
  return rc ? rc : na_status(r);
}

}  // namespace

extern "C" int jfc_solve_grid2d_noalloc(int device, void* stream, const jfc_params* params, int w, int h,
                                        const int32_t* d_excess, const int32_t* const* d_ncap,
                                        int64_t flow_offset, uint8_t* d_labels, int64_t* flow) {
  if (!d_excess || !d_ncap || !d_labels || !flow) return set_error(JFC_ERR_INVALID_ARG, "null argument");
  for (int k = 0; k < 4; ++k)
    if (!d_ncap[k]) return set_error(JFC_ERR_INVALID_ARG, "null capacity array");
  if (w < 1 || h < 1) return set_error(JFC_ERR_INVALID_ARG, "empty grid");
  const int pitch = (w + JFC_TW - 1) / JFC_TW * JFC_TW;
  const int Hp = (h + JFC_PAD_Y2 - 1) / JFC_PAD_Y2 * JFC_PAD_Y2;
  if ((long long)pitch * Hp > kMaxNodes)
    return set_error(JFC_ERR_INVALID_ARG,
                     "grid exceeds the no-allocation limit of 524288 nodes (width padded to 32, height to 16)");
  jfc_params p{};
  if (params) p = *params;
  fill_defaults(p);
  DeviceGuard restore;
  JFC_CUDA(cudaSetDevice(device));
  char* base = nullptr;
  int rc = na_scratch(device, &base);
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  const size_t plane = (size_t)pitch * Hp;

  GridDev g;
  std::memset(&g, 0, sizeof(g));
  g.dims = 2; g.W = w; g.H = h; g.D = 1;
  g.pitch = pitch; g.Hp = Hp; g.Dp = 1;
  g.plane = (long long)plane;
  g.e = (int*)(base + kOffE);
  g.h = (int*)(base + kOffH);
  for (int k = 0; k < 4; ++k) g.r[k] = (int*)(base + kOffR + k * kPlane);
  g.r[4] = g.r[5] = g.r[0];
  g.label = (uint8_t*)(base + kOffLabel);
  const int TR = p.tile_rows;
  g.tiles_x = pitch / JFC_TW;
  g.tiles_y = Hp / TR;
  g.tiles_z = 1;
  g.tile_base = 0;

  TileSet ts;
  ts.dims = 2; ts.TR = TR; ts.TY = TR; ts.TZ = 1;
  ts.ngrids = 1;
  ts.ntiles = g.tiles_x * g.tiles_y;
  ts.d_desc = (GridDev*)(base + kOffDesc);
  ts.d_info = (int4*)(base + kOffInfo);
  ts.d_flag_pr = (int*)(base + kOffFlagPr);
  for (int q = 0; q < 4; ++q) ts.d_q_pr[q >> 1][q & 1] = (int*)(base + kOffQPr + q * kTileI);
  ts.d_grid_active = (int*)(base + kOffGact);
  ts.d_grid_sum = (long long*)(base + kOffSum);
  ts.d_ctr = (DevCounters*)(base + kOffCtr);
  ts.nreg = wave_regions(g.tiles_x, Hp);
  ts.d_dirty = (uint8_t*)(base + kOffDirty);
  ts.d_vf = (uint4*)(base + kOffVf);
  ts.d_reg = (int4*)(base + kOffReg);
  ts.d_rrec = (unsigned*)(base + kOffRrec);
  ts.d_rflag[0] = (uint8_t*)(base + kOffRflag);
  ts.d_rflag[1] = (uint8_t*)(base + kOffRflag + al(kMaxReg));
  int* d_bad = (int*)(base + kOffBad);

  // ---- stage the graph: clear the planes in use, copy the caller's arrays in,
  //      zero arcs leaving the grid, clear the tables the solve reads
  for (int k = 0; k < 6; ++k) JFC_CUDA(cudaMemsetAsync(base + kOffE + k * kPlane, 0, plane * sizeof(int), s));
  JFC_CUDA(cudaMemsetAsync(g.label, 0, plane, s));
  JFC_CUDA(na_copy(g.e, d_excess, 4, w, h, pitch, Hp, false, s));
  for (int k = 0; k < 4; ++k) JFC_CUDA(na_copy(g.r[k], d_ncap[k], 4, w, h, pitch, Hp, false, s));
  JFC_CUDA(cudaMemsetAsync(d_bad, 0, sizeof(int), s));
  JFC_CUDA(launch_fix_boundary(g, 4, d_bad, s));
  JFC_CUDA(cudaMemsetAsync(base + kOffFlagPr, 0, kOffBad - kOffFlagPr, s));
  JFC_CUDA(cudaMemcpyAsync(ts.d_desc, &g, sizeof(g), cudaMemcpyHostToDevice, s));
  jfc_note_launch();
  k_na_tile_info<<<(ts.ntiles + 255) / 256, 256, 0, s>>>(ts.d_info, g.tiles_x, ts.ntiles);
  JFC_CUDA(cudaGetLastError());
  jfc_note_launch();
  k_na_regions<<<(ts.nreg + 255) / 256, 256, 0, s>>>(ts.d_reg, (g.tiles_x + JFC_WAVE_WORDS - 1) / JFC_WAVE_WORDS, ts.nreg);
  JFC_CUDA(cudaGetLastError());
  JFC_CUDA(launch_grid_sums(ts, s));
  JFC_CUDA(cudaMemcpyAsync((char*)ts.d_grid_sum + 2 * sizeof(long long), d_bad, sizeof(int), cudaMemcpyDeviceToDevice, s));
  struct { long long sums[2]; int bad; } in;
  rc = na_read(&in, ts.d_grid_sum, 2 * sizeof(long long) + sizeof(int), s);
  if (rc) return rc;
  if (in.bad) return set_error(JFC_ERR_INVALID_ARG, "negative n-link capacity");
  const long long sink_total = (long long)flow_offset - in.sums[0];  // sum ct

  // ---- solve, as engine_solve: relabels capped until no active tile is left,
  //      then exact, then the cut
  JFC_CUDA(launch_clear_counters(ts, s));
  int sweeps = 0;
  CycleState cyc{};
  cyc.h_cap = relabel_cap_for(p, 2);
  if (p.spin_limit > 0) JFC_CUDA(launch_set_limits(ts, (unsigned long long)p.spin_limit, cyc.h_cap, s));
  JFC_CUDA(launch_prepush(ts, s));
  cyc.interval0 = cyc.pr_sweeps = interval_for(p, 2);
  cyc.interval_max = p.relabel_interval_max;
  cyc.iters = cyc.iters_tail = p.local_iters;
  cyc.tail = -1;
  NaRead r;
  for (bool init = true; cyc.done != 2; init = false) {
    cyc.max_sweeps = p.max_sweeps - sweeps;
    if (!init && cyc.max_sweeps <= 0) return set_error(JFC_ERR_NOT_CONVERGED, "sweep budget exhausted");
    rc = na_run(ts, p, init, cyc, s, r);
    if (rc) return rc;
    sweeps += std::max(cyc.sweeps, 1);
  }
  if (r.ctr.cut_bad) return set_error(JFC_ERR_NOT_CONVERGED, "cut BFS reached a deficit node");
  JFC_CUDA(na_copy(g.label, d_labels, 1, w, h, pitch, Hp, true, s));
  struct { long long sums[2]; } out;
  rc = na_read(&out, ts.d_grid_sum, sizeof(out), s);
  if (rc) return rc;
  *flow = sink_total + out.sums[0];
  return JFC_OK;
}
