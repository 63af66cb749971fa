// kernels_wave.cu — 2D global relabel by bit-parallel level sets, 2D cut.
//
// Reference: graphcut_init_global_relabel / graphcut_global_relabel
// (graphcut_global_relabel.cl:19-124) driven by QGCWidget::globalRelabel
// (QGCWidget.cpp:2208-2241): heights = exact BFS distance to the deficit nodes
// (e < 0) over residual arcs.
//
// Layout.  32 neighbouring nodes of a row are one bit position each of a few
// 32-bit words ("row words").  The label plane, one byte per node, is free
// between the start of a solve and its cut, and holds eight words per row
// segment of 32 nodes in its 32 bytes:
//   0..3  residual arc +x, +y, -y, -x      4, 5  unused
//   6     deficit (e < 0)                  7     excess (e > 0)
// changed_tiles writes them, from 20 bytes per node of e and the four residual
// planes, for the tiles that something changed since the last relabel (a
// byte per tile, set by the push-relabel visits; every tile at the start of a
// solve).  All further work of a relabel is on words: 0.75 bytes per node.
//
// k_wave_relabel expands level sets: the nodes at distance d + 1 are those
// with a residual arc into a node at distance d that have no distance yet, a
// dozen word operations per 32 nodes.  A CTA takes a region of 64 rows x 6
// words together with a halo of 32 rows and one word on each side into
// registers and runs 32 levels on it with one block barrier each; what the
// halo misses from farther out cannot reach the region's interior within 32
// levels, so the interior is exact, and the interiors of all regions advance
// 32 levels per grid barrier.  Only regions that a level set can reach take
// part after the first phase.  Distances leave the words once per phase and
// node, as 128-byte row writes of the height plane.
//
// Why: the height plane's relaxation by tiles that this replaces (one CTA per
// queued 32 x 8 tile, asynchronous, after a dense pass over all planes) spent
// its time in the latency of dependent tile visits, about 7 us per 8 or 32
// nodes of distance.  A phase here takes 14 us while a few regions take part
// (load 2, 32 levels 6, heights 3, the rest and the barrier 3).  Relabels of
// one solve before / after: 15000 x 10000 RGB 37.2 / 11.5 ms, 1023 x 767 2.44
// / 1.1 ms; a solve's last ones: 15000 x 10000 1.65 / 0.43 ms, 4096 x 3072 0.46
// / 0.16 ms, 1023 x 767 0.139 / 0.045 ms.  The price is paid where all levels
// follow one narrow path: a phase costs its 10.5 us for a front of one node, so a
// corridor one node wide and 7,900 long in 120 x 130 nodes takes 2.5 ms a relabel
// instead of 1.4.
#include <algorithm>
#include <cstddef>

#include "jfc_flagbar.h"
#include "jfc_relax.cuh"

namespace {

using jfc::FULL;

constexpr int kT = JFC_WAVE_T;          // levels per phase = halo rows (<= 32, the word halo)
constexpr int kIR = JFC_WAVE_ROWS;      // interior rows of a region
constexpr int kIW = JFC_WAVE_WORDS;     // interior words of a region
constexpr int kC = kIW + 2;             // columns (words) of a region with its halo
constexpr int kS = (kIR + 2 * kT) / 4;  // strips of 4 rows
constexpr int kThreads = kC * kS;
constexpr int kList = 64;               // regions a CTA looks at in one go
static_assert(kC == 8 && kThreads == 256 && kT % 16 == 0 && kT <= 32 && kIR >= kT && kIR % 16 == 0,
              "a warp holds 8 columns x 4 strips of 4 rows");

__device__ __forceinline__ uint32_t* seg_words(const GridDev& g, int y, int c) {
  return reinterpret_cast<uint32_t*>(g.label + (long long)y * g.pitch + c * 32);
}

// Row words of the changed tiles, their heights (0 at deficits, else INF) and
// empty level-set state; the queues, flags and counters of the relabel and of the
// push-relabel phase behind it reset.  The first part of k_wave_relabel, one
// warp per changed tile; lane i of the tile's rows writes row i's words.  A
// warp looks at every nwarps-th tile, 32 at once: tiles change in clusters, and
// neighbours fall to different warps.  (As a kernel of its own, a warp for 32
// tiles in a row, it and the second launch took 15 us of every relabel of 640 x
// 480 or 1023 x 767 instead of 6.)
template <int TY>
__device__ __forceinline__ void changed_tiles(const TileSet& ts) {
  constexpr int kRows = 4;   // rows in flight: 20 loads a lane in the 64 registers that the levels leave
  DevCounters* ctr = ts.d_ctr;
  const int lane = threadIdx.x & 31;
  const long long gt = blockIdx.x * (long long)blockDim.x + threadIdx.x, gn = (long long)gridDim.x * blockDim.x;
  if (gt == 0) {
    ctr->bfs_status = 0;
    ctr->wave_q = 0;
    ctr->ticket[0] = ctr->ticket[1] = 0;
    ctr->pr_bar = 0;
    ctr->cut_bad = 0;
  }
  for (long long i = gt; i < ts.ngrids; i += gn) {
    ts.d_grid_active[i] = 0;
    ts.d_grid_sum[2 * i] = ts.d_grid_sum[2 * i + 1] = 0;
  }
  for (long long i = gt; i < ts.nreg; i += gn) ts.d_rflag[0][i] = ts.d_rflag[1][i] = 0;
  const long long nitems = ts.pr_split ? 2ll * ts.ntiles : ts.ntiles;
  for (long long i = gt; i < nitems; i += gn) ts.d_flag_pr[i] = 0;
  const long long w = gt >> 5, nw = gn >> 5;
  for (long long t0 = w; t0 < ts.ntiles; t0 += 32 * nw) {
    const long long cand = t0 + lane * nw;
    unsigned todo = __ballot_sync(FULL, cand < ts.ntiles && ts.d_dirty[cand] != 0);
    while (todo) {
      const long long tid = t0 + (__ffs(todo) - 1) * nw;
      todo &= todo - 1;
      const int4 ti = ts.d_info[tid];
      const GridDev& g = ts.d_desc[ti.x];
      const long long pitch = g.pitch;
      const int y0 = ti.z * TY;
      const long long n0 = (long long)ti.y * 32 + lane + (long long)y0 * pitch;
      uint4 arcs = make_uint4(0, 0, 0, 0), sign = make_uint4(0, 0, 0, 0);
#pragma unroll 1
      for (int j = 0; j < TY; j += kRows) {
        int e[kRows], r[4][kRows];
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
          const long long n = n0 + (j + i) * pitch;
          e[i] = g.e[n];
#pragma unroll
          for (int k = 0; k < 4; ++k) r[k][i] = g.r[k][n];
        }
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
          const unsigned xp = __ballot_sync(FULL, r[0][i] > 0), yp = __ballot_sync(FULL, r[1][i] > 0);
          const unsigned ym = __ballot_sync(FULL, r[2][i] > 0), xm = __ballot_sync(FULL, r[3][i] > 0);
          const unsigned neg = __ballot_sync(FULL, e[i] < 0), pos = __ballot_sync(FULL, e[i] > 0);
          if (lane == j + i) {
            arcs = make_uint4(xp, yp, ym, xm);
            sign = make_uint4(0, 0, neg, pos);
          }
          g.h[n0 + (j + i) * pitch] = e[i] < 0 ? 0 : JFC_INF;
        }
      }
      if (lane < TY) {
        uint4* q = reinterpret_cast<uint4*>(seg_words(g, y0 + lane, ti.y));
        q[0] = arcs;
        q[1] = sign;
        ts.d_vf[(long long)g.tile_base * TY + (long long)(y0 + lane) * g.tiles_x + ti.y] = make_uint4(0, 0, 0, 0);
      }
      if (lane == 0) ts.d_dirty[tid] = 0;
    }
  }
}

// Grid barrier number `b` (0, 1, ...) of a launch of the relabel or the cut, on a
// word whose arrivals only grow, so an arrival is also the release and nothing is
// reset.  There are two words, used by launches in turn (wave_epoch counts them;
// the launch behind finds its own zero).  The word also counts the CTAs that
// flagged a region for the next phase (FlagBar), which makes "is there a
// next phase" part of the same poll.  Bounded like jfc::grid_sync.  Returns -1 on
// error, else whether any CTA passed `any` (thread 0's) at this barrier.  dead
// (thread 0's): leave without an arrival.
__device__ __forceinline__ int wave_sync(DevCounters* ctr, unsigned epoch, unsigned b, bool any, bool dead = false) {
  __shared__ int s_res;
  __shared__ unsigned s_mine;   // (thread 0)
  __syncthreads();
  if (threadIdx.x == 0 && dead) {
    s_res = -1;
  } else if (threadIdx.x == 0) {
    unsigned long long* const bar = ctr->wave_bar + (epoch & 1u);
    unsigned mine = b == 0 ? 0u : s_mine;
    const unsigned long long add = jfc::FlagBar::arrival(b, any, mine);
    s_mine = mine;
    __threadfence();
    atomicAdd(bar, add);
    unsigned long long spins = 0, v;
    const unsigned long long cap = jfc::spin_cap(ctr);
    int res = 0;
    while (!jfc::FlagBar::complete(v = *(volatile unsigned long long*)bar, b, gridDim.x)) {
      if (jfc::vload(&ctr->error)) { res = -1; break; }
      if (++spins > cap) { atomicExch(&ctr->error, 1); res = -1; break; }
      if (spins > 16) __nanosleep(40);
    }
    __threadfence();
    if (res == 0) res = jfc::FlagBar::asked(v, b);
    s_res = res;
  }
  __syncthreads();
  return s_res;
}

// This launch's epoch: read by every CTA before its first arrival; the first CTA
// zeroes the next launch's counter, and names it behind the last barrier.
__device__ __forceinline__ unsigned wave_epoch(DevCounters* ctr) {
  const unsigned epoch = *(volatile unsigned*)&ctr->wave_epoch;
  if (blockIdx.x == 0 && threadIdx.x == 0) ctr->wave_bar[(epoch & 1u) ^ 1u] = 0;
  return epoch;
}

// What a phase writes to the height plane for one row word.
struct alignas(16) RowOut {
  unsigned got;    // nodes that got a distance (until the levels are done: that had one)
  unsigned gone;   // nodes set back to INF
  unsigned p[5];   // level within the phase, bit by bit
  unsigned pad;
};

// State of the level sets between phases, per row word: ts.d_vf = {V0, F0, V1,
// F1}, two buffers of (nodes with a distance, nodes of the last level).  A
// region rewrites the buffer that its record does not name and then names it,
// with the phase: {phase << 1 | buffer}.  A neighbour that reads the record in
// the same phase takes the other buffer, so all of a phase reads the state as
// the phase before left it.
//
// A thread holds 4 rows of one word column, a warp 16 rows x 8 words.  A level
// needs from elsewhere only edge bits (left and right words: the edge bytes of
// 4 rows packed into one shuffle each way) and edge rows (two shuffles, and
// shared memory between warps, every lane loading and storing some word so
// that no lane diverges): 6 accesses of the shared-memory pipe a warp and
// level.  The level of a node is kept as 5 bits in 5 words (P), updated two
// bits a level and three bits every four levels.  Measured per level with one
// CTA on an SM / four: 335 / 400 cycles, a chain of dependent word operations;
// whole words exchanged through shared memory 510 / 607, diverging edge lanes
// 590 / 680.
template <int TY>
__global__ void __launch_bounds__(kThreads, 4) k_wave_relabel(TileSet ts) {
  __shared__ RowOut s_out[kIR * kIW];
  __shared__ unsigned s_edge[2 * 256];                 // two buffers; see aout
  __shared__ int s_list[kList];
  __shared__ int4 s_reg[kList];
  __shared__ int s_n;
  __shared__ unsigned s_mask, s_new[2], s_tiles;
  __shared__ unsigned long long s_base;
  DevCounters* ctr = ts.d_ctr;
  if (jfc::cycle_skips(ts)) return;
  const unsigned epoch = wave_epoch(ctr);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctr->t_gr_start = jfc::global_ns();
    jfc::begin_cycle(ts);
  }
  // a wait of an earlier launch gave up (a run without a graph queues launches
  // behind it): that launch may have left arrivals in this epoch's word, so no
  // barrier would hold
  if (threadIdx.x == 0) s_tiles = (unsigned)jfc::vload(&ctr->error);
  changed_tiles<TY>(ts);
  if (wave_sync(ctr, epoch, 0, false, threadIdx.x == 0 && s_tiles != 0) < 0) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const unsigned long long t1 = jfc::global_ns();
    ctr->ns_gr_first += t1 - ctr->t_gr_start;
    ctr->t_gr_start = t1;
  }
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int c = t & (kC - 1), s = t >> 3, ws = s & 3;   // word column, strip of 4 rows, strip within the warp
  const bool inner = c >= 1 && c <= kIW && s >= kT / 4 && s < (kT + kIR) / 4;
  // edge words of a buffer: [warp + 1][first / last row][word column], zeros
  // around them; from word 192 on, what lanes without an edge store
  for (int i = t; i < 2 * 256; i += kThreads) s_edge[i] = 0;
  const int ain = ws == 0 ? (2 * warp + 1) * kC + c : ws == 3 ? 2 * (warp + 2) * kC + c : 0;
  const int aout = ws == 0 ? 2 * (warp + 1) * kC + c : ws == 3 ? (2 * (warp + 1) + 1) * kC + c : 192 + lane;
  const unsigned ml = c == 0 ? 0u : ~0u, mr = c == kC - 1 ? 0u : ~0u;
  RowOut* const mine = &s_out[inner ? (4 * (s - kT / 4)) * kIW + c - 1 : 0];   // (interior) rows kIW apart
  unsigned long long visits = 0;
  int phase = 1;
  for (;; ++phase) {
    const bool first = phase == 1;
    bool any_next = false;   // (thread 0) this CTA flagged a region for the next phase
    for (int base = blockIdx.x; base < ts.nreg; base += gridDim.x * kList) {
      // this CTA's regions of the phase (every gridDim-th, so neighbours fall
      // to different CTAs): all in the first phase, then the flagged ones
      if (t == 0) s_n = 0;
      __syncthreads();
      const long long cand = base + (long long)t * gridDim.x;
      if (t < kList && cand < ts.nreg) {
        const int4 ri = ts.d_reg[cand];   // (with the flag, not after it)
        bool take = first;
        if (!first && __ldcg(ts.d_rflag[phase & 1] + cand)) {
          ts.d_rflag[phase & 1][cand] = 0;
          take = true;
        }
        if (take) {
          const int k = atomicAdd(&s_n, 1);
          s_list[k] = (int)cand;
          s_reg[k] = ri;
        }
      }
      __syncthreads();
      const int count = s_n;
      for (int q = 0; q < count; ++q) {
        const int reg = s_list[q];
        const int4 ri = s_reg[q];   // {grid, region x, region y, first region of the grid}
        const GridDev& g = ts.d_desc[ri.x];
        const int cap = jfc::cap_of(g, ctr);
        const int level0 = (phase - 1) * kT;   // the state holds distances up to here
        const int rx = (g.tiles_x + kIW - 1) / kIW, ry = (g.Hp + kIR - 1) / kIR;
        const int wc = ri.y * kIW - 1 + c, y0 = ri.z * kIR - kT + 4 * s;
        const bool ok = wc >= 0 && wc < g.tiles_x && y0 >= 0 && y0 < g.Hp;   // (Hp is a multiple of 16)
        const long long rw = (long long)g.tile_base * TY + (long long)y0 * g.tiles_x + wc;
        if (t == 0) { s_mask = 0; s_new[0] = s_new[1] = 0; s_tiles = 0; }
        // ---- load
        uint4 arc[4];
        unsigned V[4], F[4];
        const unsigned own = __ldcg(ts.d_rrec + reg) & 1u;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          arc[i] = make_uint4(0, 0, 0, 0);
          V[i] = F[i] = 0;
        }
        if (ok) {
          unsigned rec = 0;
          if (!first) {
            const int dx = c == 0 ? -1 : c > kIW ? 1 : 0, dy = s < kT / 4 ? -1 : s >= (kT + kIR) / 4 ? 1 : 0;
            rec = __ldcg(ts.d_rrec + ri.w + (ri.z + dy) * rx + ri.y + dx);
          }
          uint4 vf[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t* w = seg_words(g, y0 + i, wc);
            arc[i] = *reinterpret_cast<const uint4*>(w);
            if (first) V[i] = w[6];
            if (!first || inner) vf[i] = __ldcg(ts.d_vf + rw + (long long)i * g.tiles_x);
          }
          const bool second = ((rec & 1u) ^ ((int)(rec >> 1) == phase ? 1u : 0u)) != 0u;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (first) {
              F[i] = V[i];
              if (inner) mine[i * kIW].gone = own ? vf[i].z : vf[i].x;   // had a distance after the last relabel
            } else {
              V[i] = second ? vf[i].z : vf[i].x;
              F[i] = second ? vf[i].w : vf[i].y;
            }
          }
        }
        if (inner) {
#pragma unroll
          for (int i = 0; i < 4; ++i) mine[i * kIW].got = V[i];
        }
        // ---- levels
        unsigned P[5][4];
#pragma unroll
        for (int b = 0; b < 5; ++b)
#pragma unroll
          for (int i = 0; i < 4; ++i) P[b][i] = 0;
        s_edge[aout] = ws < 2 ? F[0] : F[3];
        __syncthreads();
        const int dmax = min(kT, cap - 1 - level0);
#pragma unroll 1
        for (int d = 0; d < dmax; d += 4) {
          unsigned VG[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) VG[i] = V[i];
          unsigned any = 0;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int bo = (j & 1) << 8;
            const unsigned lim = d + j < dmax ? ~0u : 0u;   // (levels past the cap find nothing)
            const unsigned edge = s_edge[bo + ain];
            unsigned up = __shfl_up_sync(FULL, F[3], 8), dn = __shfl_down_sync(FULL, F[0], 8);
            // the lowest bytes of the right words' rows, the highest of the left words'
            const unsigned lo = __byte_perm(__byte_perm(F[0], F[1], 0x0040), __byte_perm(F[2], F[3], 0x0040), 0x5410);
            const unsigned hi = __byte_perm(__byte_perm(F[0], F[1], 0x0073), __byte_perm(F[2], F[3], 0x0073), 0x5410);
            const unsigned rb = __shfl_down_sync(FULL, lo, 1) & mr, lb = __shfl_up_sync(FULL, hi, 1) & ml;
            up = ws == 0 ? edge : up;
            dn = ws == 3 ? edge : dn;
            unsigned N[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              unsigned m = __funnelshift_r(F[i], rb >> (8 * i), 1) & arc[i].x;
              m |= __funnelshift_l(lb << (24 - 8 * i), F[i], 1) & arc[i].w;
              m |= (i < 3 ? F[i < 3 ? i + 1 : 3] : dn) & arc[i].y;
              m |= (i > 0 ? F[i > 0 ? i - 1 : 0] : up) & arc[i].z;
              N[i] = m & ~V[i] & lim;
            }
            s_edge[(bo ^ 256) + aout] = ws < 2 ? N[0] : N[3];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              F[i] = N[i];
              V[i] |= N[i];
              if (j & 1) P[0][i] |= N[i];
              if (j & 2) P[1][i] |= N[i];
            }
            any = N[0] | N[1] | N[2] | N[3];
            if (j < 3) __syncthreads();
          }
#pragma unroll
          for (int b = 0; b < 3; ++b) {
            const unsigned bit = 0u - ((unsigned)(d >> (2 + b)) & 1u);
#pragma unroll
            for (int i = 0; i < 4; ++i) P[2 + b][i] |= V[i] & ~VG[i] & bit;
          }
          // (the reducing barrier takes 60 cycles more than the plain one)
          if (!__syncthreads_or(any)) break;
        }
        // ---- heights of the nodes that got a distance, INF where the last
        //      relabel left one that this phase does not renew (a later phase
        //      may): a warp takes 4 row words at a time, a lane 4 columns
        unsigned pos[4] = {0, 0, 0, 0};
        unsigned got[4] = {0, 0, 0, 0};
        if (inner) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (ok) pos[i] = seg_words(g, y0 + i, wc)[7];
            RowOut o;
            got[i] = o.got = V[i] & ~mine[i * kIW].got;
            o.gone = first && ok ? mine[i * kIW].gone & ~V[i] : 0u;
#pragma unroll
            for (int b = 0; b < 5; ++b) o.p[b] = P[b][i];
            o.pad = 0;
            mine[i * kIW] = o;
          }
        }
        __syncthreads();
#pragma unroll 1
        for (int k0 = 4 * warp; k0 < kIR * kIW; k0 += 4 * (kThreads / 32)) {
          const int k = k0 + (lane >> 3), sh = 4 * (lane & 7);
          const RowOut o = s_out[k];
          const unsigned gn = (o.got >> sh) & 15u, zn = (o.gone >> sh) & 15u;
          if (!__any_sync(FULL, (gn | zn) != 0u)) continue;
          unsigned v = 0;   // the 4 columns' levels, a byte each
#pragma unroll
          for (int b = 0; b < 5; ++b) v |= ((((o.p[b] >> sh) & 15u) * 0x00204081u) & 0x01010101u) << b;
          int* h = g.h + (long long)(ri.z * kIR + k / kIW) * g.pitch + (ri.y * kIW + k % kIW) * 32 + sh;
          const int l1 = level0 + 1;
          const int4 w = make_int4(l1 + (int)(v & 255u), l1 + (int)((v >> 8) & 255u), l1 + (int)((v >> 16) & 255u),
                                   l1 + (int)(v >> 24));
          if (gn == 15u) {
            *reinterpret_cast<int4*>(h) = w;
          } else if (gn | zn) {
            if ((gn | zn) & 1u) h[0] = gn & 1u ? w.x : JFC_INF;
            if ((gn | zn) & 2u) h[1] = gn & 2u ? w.y : JFC_INF;
            if ((gn | zn) & 4u) h[2] = gn & 4u ? w.z : JFC_INF;
            if ((gn | zn) & 8u) h[3] = gn & 8u ? w.w : JFC_INF;
          }
        }
        // ---- the state, and the tiles (push-relabel items) that became active
        const bool had = !first && ((pos[0] & V[0] & ~got[0]) | (pos[1] & V[1] & ~got[1]) | (pos[2] & V[2] & ~got[2]) |
                                    (pos[3] & V[3] & ~got[3])) != 0u;
        const bool has = ((pos[0] & V[0]) | (pos[1] & V[1]) | (pos[2] & V[2]) | (pos[3] & V[3])) != 0u;
        if (inner && ok) {
          uint2* vf = reinterpret_cast<uint2*>(ts.d_vf + rw) + (own ^ 1u);
#pragma unroll
          for (int i = 0; i < 4; ++i) vf[2ll * i * g.tiles_x] = make_uint2(V[i], F[i]);
        }
        const unsigned bh = __ballot_sync(FULL, inner && had), bn = __ballot_sync(FULL, inner && has);
        // an item is 2 strips (8 rows), or 4 for whole 32 x 16 tiles
        const bool halves = TY == 8 || ts.pr_split;
        const unsigned whole = 0x01010101u << c, im = halves ? 0x101u << (lane & 23) : whole;
        const bool item_new = inner && ok && (s & (halves ? 1 : 3)) == 0 && (bn & im) && !(bh & im);
        const bool tile_new = TY == 8 ? item_new : inner && ok && ws == 0 && (bn & whole) && !(bh & whole);
        const int par = halves ? (wc + (y0 >> 3)) & 1 : (wc + (y0 >> 4)) & 1;
        int item = -1;
        if (item_new) {
          item = g.tile_base + y0 / TY * g.tiles_x + wc;
          if (TY == 16 && halves) item = 2 * item + ((y0 >> 3) & 1);
        }
        const unsigned b0 = __ballot_sync(FULL, item >= 0 && par == 0), b1 = __ballot_sync(FULL, item >= 0 && par == 1);
        const unsigned bt = __ballot_sync(FULL, tile_new);
        unsigned slot0 = 0, slot1 = 0;
        if (lane == 0) {
          if (b0) slot0 = atomicAdd(&s_new[0], __popc(b0));
          if (b1) slot1 = atomicAdd(&s_new[1], __popc(b1));
          if (bt) atomicAdd(&s_tiles, __popc(bt));
        }
        slot0 = __shfl_sync(FULL, slot0, 0) + __popc(b0 & ((1u << lane) - 1u));
        slot1 = __shfl_sync(FULL, slot1, 0) + __popc(b1 & ((1u << lane) - 1u));
        // ---- regions that the last level reaches within the next phase
        unsigned mask = 0;
        if (inner && ok && cap - 1 > level0 + kT && (F[0] | F[1] | F[2] | F[3])) {
          const int si = s - kT / 4;
          const unsigned row = (si < kT / 4 ? 1u : 0u) | 2u | (si >= (kIR - kT) / 4 ? 4u : 0u);
          const unsigned col = (c == 1 ? 1u : 0u) | 2u | (c == kIW ? 4u : 0u);
          mask = (row & 1u ? col : 0u) | (col << 3) | (row & 4u ? col << 6 : 0u);
        }
        mask = __reduce_or_sync(FULL, mask);
        if (lane == 0 && mask) atomicOr(&s_mask, mask);
        __syncthreads();
        const unsigned new0 = s_new[0], new1 = s_new[1], reach = s_mask;
        if (t == 0) {
          if (new0 | new1) s_base = atomicAdd(&ctr->wave_q, (unsigned long long)new1 << 32 | new0);
          if (s_tiles) atomicAdd(&ts.d_grid_active[ri.x], (int)s_tiles);
          any_next |= reach != 0;
          ts.d_rrec[reg] = (unsigned)phase << 1 | (own ^ 1u);
        } else if (t >= 32 && t < 41 && (reach >> (t - 32) & 1u)) {
          const int nx = ri.y + (t - 32) % 3 - 1, ny = ri.z + (t - 32) / 3 - 1;
          if (nx >= 0 && nx < rx && ny >= 0 && ny < ry) ts.d_rflag[(phase + 1) & 1][ri.w + ny * rx + nx] = 1;
        }
        if (new0 | new1) {
          __syncthreads();
          if (item >= 0) {
            ts.d_q_pr[par][0][(unsigned)(s_base >> (par ? 32 : 0)) + (par ? slot1 : slot0)] = item;
            ts.d_flag_pr[item] = 1;
          }
        }
        ++visits;
        __syncthreads();   // the shared state is free for the next region
      }
    }
    if (wave_sync(ctr, epoch, phase, any_next) <= 0) break;
  }
  if (t == 0) {
    atomicAdd(&ctr->bfs_visits, visits * (unsigned long long)(kIR / TY * kIW));
    if (blockIdx.x == 0) {
      // (behind the last barrier: every append is counted)
      const unsigned long long q = *(volatile unsigned long long*)&ctr->wave_q;
      ctr->qn_pr[0][0] = (int)(unsigned)q;
      ctr->qn_pr[1][0] = (int)(q >> 32);
      ctr->qn_pr[0][1] = ctr->qn_pr[1][1] = 0;
      ctr->cur_pr[0] = ctr->cur_pr[1] = 0;
      ctr->bfs_passes = phase;
      ctr->bfs_status = 1;
      ctr->wave_epoch = epoch + 1;
      ctr->ns_gr_frontier += jfc::global_ns() - ctr->t_gr_start;
    }
  }
  if (blockIdx.x == 0 && warp == 0) jfc::end_cycle(ts);
}

// Cut (graphcut_init_cut / graphcut_compute_cut, graphcut_compute_cut.cl:19-140):
// the source side is every node reachable from {e > 0} along residual arcs;
// reaching a deficit raises cut_bad (the reference's done[1] divergence flag).
// On the row words that the last global relabel left in the label plane, with
// the same regions and threads: a region and its halo run to their fixpoint (a
// step closes every word, moves down and up the thread's 4 rows and across
// the edges), the interior's reached nodes go to ts.d_vf (.x of a row word; only
// their owner writes them and they only grow, so a neighbour may read them at
// any time), and a neighbour whose border an arc from a newly reached node
// crosses takes part in the next phase.  A last pass writes the label bytes
// over the words and sums min(e, 0) and the labels per grid.  Every region's
// first visit reads 1 byte per node; the tile-wise pass over e and the arcs (21
// bytes per node, and one warp for 32 tiles in turn) and the separate sums took
// 0.22 ms on 640 x 480 and 2.1 ms on 15000 x 10000, this 0.042 and 0.46 (of
// which 0.12 are the excess and label planes at the HBM rate).
template <int TY>
__global__ void __launch_bounds__(kThreads, 4) k_wave_cut(TileSet ts, int max_passes) {
  __shared__ unsigned s_edge[2 * 256];   // as in k_wave_relabel
  __shared__ int s_list[kList];
  __shared__ int4 s_reg[kList];
  __shared__ int s_n;
  __shared__ unsigned s_mask;
  __shared__ long long s_sum[2][kThreads / 32];
  DevCounters* ctr = ts.d_ctr;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int c = t & (kC - 1), s = t >> 3, ws = s & 3;
  const bool inner = c >= 1 && c <= kIW && s >= kT / 4 && s < (kT + kIR) / 4;
  for (int i = t; i < 2 * 256; i += kThreads) s_edge[i] = 0;
  const int ain = ws == 0 ? (2 * warp + 1) * kC + c : ws == 3 ? 2 * (warp + 2) * kC + c : 0;
  const int aout = ws == 0 ? 2 * (warp + 1) * kC + c : ws == 3 ? (2 * (warp + 1) + 1) * kC + c : 192 + lane;
  const unsigned ml = c == 0 ? 0u : ~0u, mr = c == kC - 1 ? 0u : ~0u;
  unsigned long long visits = 0;
  if (jfc::cycle_skips(ts)) return;
  const unsigned epoch = wave_epoch(ctr);
  if (blockIdx.x == 0 && t == 0) ctr->t_gr_start = jfc::global_ns();
  int phase = 1;
  bool ok_all = true;
  for (;; ++phase) {
    const bool first = phase == 1;
    bool any_next = false;   // (thread 0) this CTA flagged a region for the next phase
    for (int base = blockIdx.x; base < ts.nreg; base += gridDim.x * kList) {
      if (t == 0) s_n = 0;
      __syncthreads();
      const long long cand = base + (long long)t * gridDim.x;
      if (t < kList && cand < ts.nreg) {
        const int4 ri = ts.d_reg[cand];
        bool take = first;
        if (!first && __ldcg(ts.d_rflag[phase & 1] + cand)) {
          ts.d_rflag[phase & 1][cand] = 0;
          take = true;
        }
        if (take) {
          const int k = atomicAdd(&s_n, 1);
          s_list[k] = (int)cand;
          s_reg[k] = ri;
        }
      }
      __syncthreads();
      const int count = s_n;
      for (int q = 0; q < count; ++q) {
        const int4 ri = s_reg[q];
        const GridDev& g = ts.d_desc[ri.x];
        const int rx = (g.tiles_x + kIW - 1) / kIW, ry = (g.Hp + kIR - 1) / kIR;
        const int wc = ri.y * kIW - 1 + c, y0 = ri.z * kIR - kT + 4 * s;
        const bool ok = wc >= 0 && wc < g.tiles_x && y0 >= 0 && y0 < g.Hp;
        const long long rw = (long long)g.tile_base * TY + (long long)y0 * g.tiles_x + wc;
        if (t == 0) s_mask = 0;
        uint4 arc[4];
        unsigned L[4], L0[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          arc[i] = make_uint4(0, 0, 0, 0);
          L[i] = 0;
          if (ok) {
            const uint32_t* w = seg_words(g, y0 + i, wc);
            arc[i] = *reinterpret_cast<const uint4*>(w);
            L[i] = first ? w[7] : __ldcg(&ts.d_vf[rw + (long long)i * g.tiles_x].x);
          }
          L0[i] = L[i];
        }
        auto publish = [&](int bo) { s_edge[bo + aout] = ws < 2 ? L[0] & arc[0].z : L[3] & arc[3].y; };
        publish(0);
        __syncthreads();
        bool fresh = true;   // the words are not closed yet
        for (int step = 0;; ++step) {
          const int bo = (step & 1) << 8;
          const unsigned edge = s_edge[bo + ain];
          unsigned up = __shfl_up_sync(FULL, L[3] & arc[3].y, 8), dn = __shfl_down_sync(FULL, L[0] & arc[0].z, 8);
          unsigned lo = 0, hi = 0;   // bit i: row i's word sends to the left / right word
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            lo |= (L[i] & arc[i].w & 1u) << i;
            hi |= ((L[i] & arc[i].x) >> 31) << i;
          }
          const unsigned rb = __shfl_down_sync(FULL, lo, 1) & mr, lb = __shfl_up_sync(FULL, hi, 1) & ml;
          up = ws == 0 ? edge : up;
          dn = ws == 3 ? edge : dn;
          unsigned came = 0;
          const unsigned was[4] = {L[0], L[1], L[2], L[3]};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const unsigned in = (lb >> i & 1u) | (rb >> i & 1u) << 31 | (i == 0 ? up : 0u) | (i == 3 ? dn : 0u);
            came |= in & ~L[i];
            L[i] |= in;
          }
          if (__any_sync(FULL, came != 0u || fresh)) {
#pragma unroll
            for (int turn = 0; turn < 2; ++turn) {
#pragma unroll
              for (int i = 0; i < 4; ++i) L[i] = jfc::close_left(jfc::close_right(L[i], arc[i].x << 1), arc[i].w >> 1);
#pragma unroll
              for (int i = 1; i < 4; ++i) L[i] |= L[i - 1] & arc[i - 1].y;
#pragma unroll
              for (int i = 2; i >= 0; --i) L[i] |= L[i + 1] & arc[i + 1].z;
            }
            // not closed if the last moves across rows left something to close
            bool open = false;
#pragma unroll
            for (int i = 0; i < 4; ++i)
              open |= (((L[i] & arc[i].x) << 1 | (L[i] & arc[i].w) >> 1) & ~L[i]) != 0u;
            fresh = open;
          }
          publish(bo ^ 256);
          // (what changed in this step has to reach the neighbours in the next)
          if (!__syncthreads_or(fresh || ((L[0] ^ was[0]) | (L[1] ^ was[1]) | (L[2] ^ was[2]) | (L[3] ^ was[3])) != 0u)) break;
        }
        // ---- the interior's reached nodes, and the neighbours they reach
        unsigned mask = 0;
        bool hit = false;
        if (inner && ok) {
          unsigned news[4], any = 0;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            news[i] = L[i] & ~L0[i];
            any |= news[i];
          }
          if (first || any) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              ts.d_vf[rw + (long long)i * g.tiles_x].x = L[i];
              hit |= (L[i] & seg_words(g, y0 + i, wc)[6]) != 0u;
            }
          }
          unsigned left = 0, right = 0;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            left |= news[i] & arc[i].w & 1u;
            right |= (news[i] & arc[i].x) >> 31;
          }
          if (s == kT / 4 && (news[0] & arc[0].z)) mask |= 1u;
          if (s == (kT + kIR) / 4 - 1 && (news[3] & arc[3].y)) mask |= 2u;
          if (c == 1 && left) mask |= 4u;
          if (c == kIW && right) mask |= 8u;
        }
        if (hit) *(volatile int*)&ctr->cut_bad = 1;
        mask = __reduce_or_sync(FULL, mask);
        if (lane == 0 && mask) atomicOr(&s_mask, mask);
        __syncthreads();
        const unsigned reach = s_mask;
        if (t == 0) any_next |= reach != 0;
        if (t < 4 && (reach >> t & 1u)) {
          const int nx = ri.y + (t == 2 ? -1 : t == 3 ? 1 : 0), ny = ri.z + (t == 0 ? -1 : t == 1 ? 1 : 0);
          if (nx >= 0 && nx < rx && ny >= 0 && ny < ry) ts.d_rflag[(phase + 1) & 1][ri.w + ny * rx + nx] = 1;
        }
        ++visits;
        __syncthreads();
      }
    }
    const int more = wave_sync(ctr, epoch, phase - 1, any_next);
    if (more < 0) ok_all = false;
    if (more <= 0) break;
    if (phase > max_passes) {
      if (blockIdx.x == 0 && t == 0) ctr->bfs_status = 2;
      ok_all = false;
      break;
    }
  }
  // ---- labels and sums: a region's words, 8 lanes per row word, 4 nodes a lane
  if (ok_all) {
    for (int reg = blockIdx.x; reg < ts.nreg; reg += gridDim.x) {
      const int4 ri = ts.d_reg[reg];
      const GridDev& g = ts.d_desc[ri.x];
      long long neg = 0, lab = 0;
      for (int k = t >> 3; k < kIR * kIW; k += kThreads / 8) {
        const int y = ri.z * kIR + k / kIW, w = ri.y * kIW + k % kIW, sh = 4 * (t & 7);
        if (y >= g.Hp || w >= g.tiles_x) continue;
        const unsigned L = __ldcg(&ts.d_vf[(long long)g.tile_base * TY + (long long)y * g.tiles_x + w].x);
        const unsigned nib = (L >> sh) & 15u;
        const long long n = (long long)y * g.pitch + w * 32 + sh;
        const int4 e = *reinterpret_cast<const int4*>(g.e + n);
        *reinterpret_cast<unsigned*>(g.label + n) = (nib * 0x00204081u) & 0x01010101u;
        neg += (long long)min(e.x, 0) + min(e.y, 0) + min(e.z, 0) + min(e.w, 0);
        lab += __popc(nib);
      }
      for (int o = 16; o; o >>= 1) {
        neg += __shfl_xor_sync(FULL, neg, o);
        lab += __shfl_xor_sync(FULL, lab, o);
      }
      if (lane == 0) {
        s_sum[0][warp] = neg;
        s_sum[1][warp] = lab;
      }
      __syncthreads();
      if (t < 2) {
        long long v = 0;
        for (int w = 0; w < kThreads / 32; ++w) v += s_sum[t][w];
        atomicAdd((unsigned long long*)&ts.d_grid_sum[2 * ri.x + t], (unsigned long long)v);
      }
      __syncthreads();
    }
  }
  if (t == 0) {
    atomicAdd(&ctr->bfs_visits, visits * (unsigned long long)(kIR / TY * kIW));
    if (blockIdx.x == 0) {
      ctr->bfs_passes = phase;
      ctr->wave_epoch = epoch + 1;
      ctr->ns_cut = jfc::global_ns() - ctr->t_gr_start;
      if (ok_all) ctr->bfs_status = 1;
    }
  }
}

template <int TY>
cudaError_t wave_cut_t(const TileSet& ts, int max_passes, cudaStream_t s) {
  static int cache[64] = {0};
  const void* fn = (const void*)k_wave_cut<TY>;
  // (in a run of cycles the relabel before it cleared them, and may have set the status)
  cudaError_t e = ts.cyc_mode ? cudaSuccess : cudaMemsetAsync(ts.d_grid_sum, 0, sizeof(long long) * 2 * ts.ngrids, s);
  static_assert(offsetof(DevCounters, bfs_status) == offsetof(DevCounters, cut_bad) + sizeof(int), "zeroed together");
  if (e == cudaSuccess && !ts.cyc_mode) e = cudaMemsetAsync(&ts.d_ctr->cut_bad, 0, 2 * sizeof(int), s);
  if (e != cudaSuccess) return e;
  const int blocks = std::min({persistent_blocks_cached(cache, fn, kThreads), ts.nreg, (int)jfc::kFlagBarBlocks});
  TileSet arg = ts;
  void* params[] = {(void*)&arg, (void*)&max_passes};
  jfc_note_launch();
  return cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(kThreads), params, 0, s);
}

template <int TY>
cudaError_t wave_t(const TileSet& ts, cudaStream_t s) {
  static int cache[64] = {0};
  const void* fn = (const void*)k_wave_relabel<TY>;
  // no more CTAs than regions: the grid barrier's cost grows with them
  const int blocks = std::min({persistent_blocks_cached(cache, fn, kThreads), ts.nreg, (int)jfc::kFlagBarBlocks});
  TileSet arg = ts;
  void* params[] = {(void*)&arg};
  jfc_note_launch();
  return cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(kThreads), params, 0, s);
}

}  // namespace

cudaError_t launch_wave_relabel(const TileSet& ts, cudaStream_t s) {
  if (ts.ntiles <= 0) return cudaSuccess;
  if (ts.TR == 8) return wave_t<8>(ts, s);
  if (ts.TR == 16) return wave_t<16>(ts, s);
  return cudaErrorInvalidValue;
}

cudaError_t launch_wave_cut(const TileSet& ts, int max_passes, cudaStream_t s) {
  if (ts.ntiles <= 0) return cudaSuccess;
  if (ts.TR == 8) return wave_cut_t<8>(ts, max_passes, s);
  if (ts.TR == 16) return wave_cut_t<16>(ts, max_passes, s);
  return cudaErrorInvalidValue;
}
