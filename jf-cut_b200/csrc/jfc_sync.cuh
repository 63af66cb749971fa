// jfc_sync.cuh — device work queues and the grid barrier of the persistent
// (cooperative) phase kernels.
#pragma once

#include "jfc_internal.h"

namespace jfc {

constexpr unsigned FULL = 0xffffffffu;

// Polls a device-side wait makes before it gives up: ctr->spin_limit, or
// 2^26 (seconds) when it is 0.
__device__ __forceinline__ unsigned long long spin_cap(const DevCounters* ctr) {
  const unsigned long long v = *(const volatile unsigned long long*)&ctr->spin_limit;
  return v ? v : (1ull << 26);
}

// Grid-wide barrier of a cooperative launch.  Every wait is bounded: after
// spin_cap polls the barrier raises ctr->error and returns false, and every
// block leaves its loop on the next check, so a lost block can never hang
// the device.  `on_last` runs on the last block to arrive, before the
// release (queue / ticket resets between phases).
template <typename F>
__device__ __forceinline__ bool grid_sync(DevCounters* ctr, F on_last) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned* vgen = &ctr->bar_gen;
    volatile int* verr = &ctr->error;
    const unsigned g = *vgen;
    __threadfence();
    int ok = 1;
    if (atomicAdd(&ctr->bar_count, 1u) == gridDim.x - 1) {
      on_last();
      ctr->bar_count = 0;
      __threadfence();
      atomicAdd(&ctr->bar_gen, 1u);
    } else {
      unsigned long long spins = 0;
      const unsigned long long cap = spin_cap(ctr);
      while (*vgen == g) {
        if (*verr) { ok = 0; break; }
        if (++spins > cap) { atomicExch(&ctr->error, 1); ok = 0; break; }
        __nanosleep(100);
      }
    }
    __threadfence();
    s_ok = ok && (*verr == 0);
  }
  __syncthreads();
  return s_ok != 0;
}

__device__ __forceinline__ int vload(const int* p) { return *(const volatile int*)p; }

// Grid barrier on a counter that only grows (zero at the kernel's start): an
// arrival is also the release, so the waiting is one atomic and one poll, 1.6
// us against 3 us of grid_sync with its generation word and its reset by the
// last block.  `target`: blocks x barriers so far.  Bounded like grid_sync.
__device__ __forceinline__ bool arrive_wait(DevCounters* ctr, unsigned long long* counter, unsigned long long target) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(counter, 1ull);
    unsigned long long spins = 0;
    const unsigned long long cap = spin_cap(ctr);
    int ok = 1;
    while (*(volatile unsigned long long*)counter < target) {
      if (vload(&ctr->error)) { ok = 0; break; }
      if (++spins > cap) { atomicExch(&ctr->error, 1); ok = 0; break; }
      if (spins > 8) __nanosleep(64);
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// Distance cap of the running global relabel: distances at or above it are
// stored as unreachable (JFC_INF); no cap when ctr->cyc.h_cap is 0.
// (set before the kernel that reads it runs, constant during it: an ordinary
// cached load, not a poll of L2 on every tile visit)
__device__ __forceinline__ int height_cap(const DevCounters* ctr) {
  const int v = ctr->cyc.h_cap;
  return v > 0 ? v : JFC_INF;
}
// The cap for grid g: its own when set, else the tile set's.
__device__ __forceinline__ int cap_of(const GridDev& g, const DevCounters* ctr) {
  return g.h_cap > 0 ? g.h_cap : height_cap(ctr);
}

// Device-wide nanosecond clock (phase timing of the persistent kernels).
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// A launch of a run of cycles that is not due (the same for all of its CTAs: only
// a relabel's end changes it).
__device__ __forceinline__ bool cycle_skips(const TileSet& ts) {
  const CycleState& c = ts.d_ctr->cyc;
  return ts.cyc_mode == 2 ? !vload(&c.go) : ts.cyc_mode == 3 ? vload(&c.done) != 1
       : ts.cyc_mode == 4 ? vload(&c.done) != 2 : false;
}

// A loop that this relabel ends a turn of stops unless end_cycle says otherwise
// (one thread, at the relabel's start: a relabel that gives up ends the loop).
__device__ __forceinline__ void begin_cycle(const TileSet& ts) {
  if (ts.cyc_cond) cudaGraphSetConditional((cudaGraphConditionalHandle)ts.cyc_cond, 0u);
}

// End of a relabel cycle, one warp, behind the relabel's last barrier and its
// thread 0's counters: advance the schedule, and let the loop go on while tiles
// are active and no limit is reached.  Without active tiles under the cap the
// exact relabel is due, without any the cut: both are behind the loop in the
// same run.  A cycle decided by the host costs 28 us
// besides its kernels (read-back, wait, launch), a turn of the graph's loop 10
// (1023 x 767: 14 relabels, 2.12 / 1.94 ms).
__device__ __forceinline__ void end_cycle(const TileSet& ts) {
  if (ts.cyc_mode == 0) return;
  DevCounters* ctr = ts.d_ctr;
  const int lane = threadIdx.x & 31;
  long long active = 0;
  for (int i = lane; i < ts.ngrids; i += 32) active += __ldcg(ts.d_grid_active + i);
  for (int o = 16; o; o >>= 1) active += __shfl_xor_sync(FULL, active, o);
  if (lane != 0) return;
  CycleState c = ctr->cyc;
  const bool tail = cycle_tail(active, ts.ntiles);
  const unsigned long long gr = ctr->ns_gr_first + ctr->ns_gr_frontier, pr = ctr->ns_pr;
  if (ts.cyc_mode == 2) {
    const int sw = ctr->sweeps_done;
    c.pr_sweeps = next_interval(c, tail, pr - c.last_pr, gr - c.last_gr, sw);
    c.sweeps += sw;
  }
  c.local_iters = tail ? c.iters_tail : c.iters;
  c.last_pr = pr;
  c.last_gr = gr;
  c.cycles += 1;
  c.passes += ctr->bfs_passes;
  const bool ok = vload(&ctr->error) == 0 && ctr->bfs_status == 1;
  c.go = ok && ts.cyc_mode != 3 && active > 0 && c.cycles < c.max_cycles && c.sweeps < c.max_sweeps &&
         (c.tail < 0 || (c.tail != 0) == tail);
  c.done = ok && active == 0 ? (c.h_cap > 0 ? 1 : 2) : 0;
  if (ts.cyc_mode == 3) c.exact += 1;
  if (c.done == 1) c.h_cap = 0;
  ctr->cyc = c;
  if (c.go && ts.cyc_cond) cudaGraphSetConditional((cudaGraphConditionalHandle)ts.cyc_cond, 1u);
}

// Phase-clock instrumentation (builds with -DJFC_PHASE_CLOCK): thread 0 adds
// the SM cycles since `t` to counter k and restarts `t`.
#ifdef JFC_PHASE_CLOCK
#define JFC_PCLK_DECL long long _pclk = clock64();
#define JFC_PCLK(ctr, k)                                                            \
  do {                                                                              \
    if (threadIdx.x == 0) {                                                         \
      const long long _n = clock64();                                               \
      atomicAdd(&(ctr)->prof[k], (unsigned long long)(_n - _pclk));                 \
      _pclk = _n;                                                                   \
    }                                                                               \
  } while (0)
#else
#define JFC_PCLK_DECL
#define JFC_PCLK(ctr, k) do {} while (0)
#endif

// Warp-cooperative append of up to 32 candidate tiles: lane k offers `tile`
// when `want`; with `flags`, a tile is appended only by the lane that flips
// its flag 0 -> 1 (so a queue never holds a tile twice).
__device__ __forceinline__ void warp_append(bool want, int tile, int* flags, int* queue, int* qn) {
  bool won = false;
  if (want) won = flags ? (atomicExch(flags + tile, 1) == 0) : true;
  const unsigned m = __ballot_sync(FULL, won);
  if (!m) return;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(m) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(qn, __popc(m));
  base = __shfl_sync(FULL, base, leader);
  if (won) queue[base + __popc(m & ((1u << lane) - 1u))] = tile;
}

// One warp-level ticket from a device counter.
__device__ __forceinline__ unsigned warp_ticket(unsigned* t) {
  unsigned v = 0;
  if ((threadIdx.x & 31) == 0) v = atomicAdd(t, 1u);
  return __shfl_sync(FULL, v, 0);
}

}  // namespace jfc
