// kernels_bfs.cu — 3D global relabel and cut, tag BFS, reductions and layout
// helpers (the 2D relabel and cut: kernels_wave.cu).
//
// Global relabel — reference graphcut_init_global_relabel / graphcut_global_relabel
// (graphcut_global_relabel.cl:128-249) driven by QGCWidget::globalRelabel
// (QGCWidget.cpp:2208-2241): heights = exact BFS distance to the deficit nodes
// (e < 0) over residual arcs, by in-tile fixpoint relaxation with tiles
// revisited in level sweeps ordered by the jump-flooding tile BFS
// (graphcut_bfs_block.cl).  Here the relaxation is monotone (heights only fall
// from INF), so tiles need no parity and no order: a first pass over every
// tile (bit-parallel level BFS on row words), then a persistent cooperative
// kernel drains the frontier (a tile whose boundary fell queues its
// neighbours) in passes separated by grid barriers, one warp per queued tile.
// Each visit records whether the tile holds an active node (e > 0, h < INF):
// the device-side active-tile count (graphcut_count_node,
// graphcut_count_block.cl:19-47) that decides convergence, and the queue of
// tiles the next push-relabel phase visits.
#include <algorithm>

#include "jfc_relax.cuh"
#include "jfc_tma.cuh"

namespace {

using jfc::FULL;

// Frontier the tile visits feed (next pass), deduplicated by its flags.
struct BfsQ {
  int* flags;
  int* q;
  int* qn;
  // staging in shared memory (null: appends go straight to the queue): the
  // items that won their flag are collected in sbuf (count *scnt) and the
  // caller moves them to the queue with one counter update per batch, so
  // thousands of warps do not all serialise on the queue's one counter
  // (the warp form of the 3D frontier passes)
  int* sbuf = nullptr;
  int* scnt = nullptr;
};

// Move a warp's staged items of Q to its queue with one counter update (all
// lanes, after a __syncwarp; the caller resets the count).
__device__ __forceinline__ void flush_staged(const BfsQ& Q, int lane) {
  const int cnt = *(volatile int*)Q.scnt;
  if (cnt == 0) return;
  int base = 0;
  if (lane == 0) base = atomicAdd(Q.qn, cnt);
  base = __shfl_sync(FULL, base, 0);
  for (int i = lane; i < cnt; i += 32) Q.q[base + i] = Q.sbuf[i];
}

struct Addr {
  long long base, pitch, slab;
  bool has_yT, has_yB, has_zT, has_zB, has_xL, has_xR;
  int x0, y0, z0;
};

template <int DIMS, int TY, int TZ>
__device__ __forceinline__ Addr make_addr(const GridDev& g, int4 ti, int lane) {
  Addr a;
  a.pitch = g.pitch;
  a.slab = (long long)g.pitch * g.Hp;
  a.x0 = ti.y * 32; a.y0 = ti.z * TY; a.z0 = ti.w * TZ;
  a.base = (long long)(a.x0 + lane) + (long long)a.y0 * a.pitch + (long long)a.z0 * a.slab;
  a.has_yT = a.y0 > 0;
  a.has_yB = a.y0 + TY < g.Hp;
  a.has_zT = (DIMS == 3) && a.z0 > 0;
  a.has_zB = (DIMS == 3) && (a.z0 + TZ < g.Dp);
  a.has_xL = a.x0 > 0;
  a.has_xR = a.x0 + 32 < g.pitch;
  return a;
}

template <int TY>
__device__ __forceinline__ long long roff(const Addr& a, int i) {
  return a.base + (long long)(i % TY) * a.pitch + (long long)(i / TY) * a.slab;
}

// Queue the neighbour tiles whose halo changed (rows_changed: rows of this
// tile that changed; c0 / c31: a change in the first / last column) and the
// tile itself when its in-tile fixpoint is not reached yet.
template <int DIMS, int TY, int TZ>
__device__ __forceinline__ void flag_neighbours(const GridDev& g, const Addr& a, int tid, unsigned rows_changed,
                                                bool c0, bool c31, bool again, const BfsQ& Q) {
  const int lane = threadIdx.x & 31;
  unsigned ymask0 = 0, ymask1 = 0, zmask0 = 0, zmask1 = 0;
#pragma unroll
  for (int z = 0; z < TZ; ++z) { ymask0 |= 1u << (z * TY); ymask1 |= 1u << (z * TY + TY - 1); }
#pragma unroll
  for (int y = 0; y < TY; ++y) { zmask0 |= 1u << y; zmask1 |= 1u << ((TZ - 1) * TY + y); }
  const int txs = g.tiles_x, tys = g.tiles_y;
  bool want = false;
  int nb = tid;
  switch (lane) {
    case 0: want = (rows_changed & ymask0) && a.has_yT; nb = tid - txs; break;
    case 1: want = (rows_changed & ymask1) && a.has_yB; nb = tid + txs; break;
    case 2: want = c0 && a.has_xL; nb = tid - 1; break;
    case 3: want = c31 && a.has_xR; nb = tid + 1; break;
    case 4: want = DIMS == 3 && (rows_changed & zmask0) && a.has_zT; nb = tid - txs * tys; break;
    case 5: want = DIMS == 3 && (rows_changed & zmask1) && a.has_zB; nb = tid + txs * tys; break;
    case 6: want = again; nb = tid; break;
    default: break;
  }
  if (Q.sbuf) {
    if (want && atomicExch(Q.flags + nb, 1) == 0) Q.sbuf[atomicAdd(Q.scnt, 1)] = nb;
  } else {
    jfc::warp_append(want, nb, Q.flags, Q.q, Q.qn);
  }
}

// ------------------------------------------------------------------ tag BFS
// The reference's tag post-process (graphcut_compute_tag.cl): reachability from
// the foreground seeds through object nodes (any direction), kept in bit 1 of
// the label byte; `seeds` is the dense seed array (JFC_SEED_FG = 1).  One warp
// per tile: R rows of 32-bit words (bit = lane), row closure by 5-step shift
// doubling, rows combined by word AND / OR.
template <int DIMS, int TY, int TZ, bool FIRST>
__device__ __forceinline__ void tag_tile(const GridDev& g, int4 ti, int tid, const BfsQ& Q,
                                         const uint8_t* __restrict__ seeds) {
  constexpr int R = TY * TZ;
  const int lane = threadIdx.x & 31;
  const Addr a = make_addr<DIMS, TY, TZ>(g, ti, lane);
  uint8_t* __restrict__ Lb = g.label;
  unsigned L[R], L0[R], OBJ[R];   // tagged nodes, object nodes
  auto is_seed = [&](int x, int y, int z) -> bool {
    return x < g.W && y < g.H && z < g.D && seeds[x + (long long)g.W * (y + (long long)g.H * z)] == JFC_SEED_FG;
  };
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const unsigned lb = Lb[roff<TY>(a, i)];
    OBJ[i] = __ballot_sync(FULL, lb & 1u);
    if constexpr (FIRST) L[i] = __ballot_sync(FULL, is_seed(a.x0 + lane, a.y0 + i % TY, a.z0 + i / TY));
    else L[i] = __ballot_sync(FULL, (lb & 2u) != 0);
    L0[i] = L[i];
  }
  // a tagged node of the halo (an object node beside it takes the tag)
  auto halo_tag = [&](long long n) -> bool {
    if constexpr (FIRST) {
      const long long yz = n / g.pitch;
      return is_seed((int)(n % g.pitch), (int)(yz % g.Hp), (int)(yz / g.Hp));
    } else {
      return (Lb[n] & 2u) != 0;
    }
  };
#pragma unroll
  for (int z = 0; z < TZ; ++z) {
    const long long n = roff<TY>(a, z * TY);
    L[z * TY] |= __ballot_sync(FULL, a.has_yT && halo_tag(n - a.pitch)) & OBJ[z * TY];
    L[z * TY + TY - 1] |= __ballot_sync(FULL, a.has_yB && halo_tag(n + (long long)TY * a.pitch)) & OBJ[z * TY + TY - 1];
  }
  if constexpr (DIMS == 3) {
#pragma unroll
    for (int y = 0; y < TY; ++y) {
      const long long n = roff<TY>(a, y);
      L[y] |= __ballot_sync(FULL, a.has_zT && halo_tag(n - a.slab)) & OBJ[y];
      L[(TZ - 1) * TY + y] |= __ballot_sync(FULL, a.has_zB && halo_tag(n + (long long)TZ * a.slab)) & OBJ[(TZ - 1) * TY + y];
    }
  }
  {
    const int row = lane & 15;
    const bool left = lane < 16;
    bool s = false;
    if (row < R && (left ? a.has_xL : a.has_xR))
      s = halo_tag((long long)(left ? a.x0 - 1 : a.x0 + 32) + (long long)(a.y0 + row % TY) * a.pitch +
                   (long long)(a.z0 + row / TY) * a.slab);
    const unsigned sb = __ballot_sync(FULL, s);
#pragma unroll
    for (int i = 0; i < R; ++i) L[i] |= ((sb >> i & 1u) | (sb >> (16 + i) & 1u) << 31) & OBJ[i];
  }
  bool converged = false;
  for (int it = 0; it < 64; ++it) {
    unsigned ch = 0;
    auto grow = [&](int i, unsigned p) { ch |= p ^ L[i]; L[i] = p; };
#pragma unroll
    for (int i = 0; i < R; ++i) grow(i, jfc::close_left(jfc::close_right(L[i], OBJ[i] & ~1u), OBJ[i] & 0x7fffffffu));
#pragma unroll
    for (int i = 1; i < R; ++i) if (i % TY > 0) grow(i, L[i] | (L[i - 1] & OBJ[i]));
#pragma unroll
    for (int i = R - 2; i >= 0; --i) if (i % TY < TY - 1) grow(i, L[i] | (L[i + 1] & OBJ[i]));
    if constexpr (DIMS == 3) {
#pragma unroll
      for (int i = TY; i < R; ++i) grow(i, L[i] | (L[i - TY] & OBJ[i]));
#pragma unroll
      for (int i = R - TY - 1; i >= 0; --i) grow(i, L[i] | (L[i + TY] & OBJ[i]));
    }
    if (!ch) { converged = true; break; }
  }
  unsigned rows_changed = 0, col0 = 0, col31 = 0;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const unsigned c = L[i] ^ L0[i];
    if (c) rows_changed |= 1u << i;
    col0 |= c & 1u;
    col31 |= c >> 31;
    if (FIRST || c) {
      uint8_t* p = Lb + roff<TY>(a, i);
      *p = (uint8_t)((*p & 1u) | (((L[i] >> lane) & 1u) << 1));
    }
  }
  // boundary tags that differ from what the neighbours last read
  flag_neighbours<DIMS, TY, TZ>(g, a, tid, rows_changed, col0 != 0, col31 != 0, !converged, Q);
}

// Persistent tag BFS: pass 0 visits every tile (tags start at the seeds), later
// passes drain the frontier built by the previous one (one tile per warp
// ticket), grid barriers in between, until a pass queues nothing or the pass
// budget runs out.
template <int DIMS, int TY, int TZ>
__global__ void __launch_bounds__(256) k_tag(TileSet ts, int max_passes, const uint8_t* seeds) {
  DevCounters* ctr = ts.d_ctr;
  const int lane = threadIdx.x & 31;
  unsigned long long visits = 0;
  bool ok = true;
  int pass = 0;
  {
    BfsQ Q{ts.d_flag_bfs[1], ts.d_q_bfs[1], &ctr->qn_bfs[1]};
    for (;;) {
      const unsigned c = jfc::warp_ticket(&ctr->ticket[0]);
      const long long b = (long long)c * 32;
      if (b >= ts.ntiles) break;
      const int cnt = (int)min(32ll, (long long)ts.ntiles - b);
      for (int k = 0; k < cnt; ++k) {
        const int tt = (int)b + k;
        const int4 ti = ts.d_info[tt];
        tag_tile<DIMS, TY, TZ, true>(ts.d_desc[ti.x], ti, tt, Q, seeds);
        ++visits;
      }
    }
    ok = jfc::grid_sync(ctr, [&]() { ctr->ticket[0] = 0; });
  }
  for (pass = 1; ok; ++pass) {
    const int cb = pass & 1;
    const int n = jfc::vload(&ctr->qn_bfs[cb]);
    if (n == 0) break;
    if (pass > max_passes) {
      if (blockIdx.x == 0 && threadIdx.x == 0) ctr->bfs_status = 2;
      break;
    }
    BfsQ Q{ts.d_flag_bfs[cb ^ 1], ts.d_q_bfs[cb ^ 1], &ctr->qn_bfs[cb ^ 1]};
    const int* queue = ts.d_q_bfs[cb];
    int* fcur = ts.d_flag_bfs[cb];
    for (;;) {
      const unsigned k = jfc::warp_ticket(&ctr->ticket[cb]);
      if ((int)k >= n) break;
      const int tt = queue[k];
      if (lane == 0) fcur[tt] = 0;
      __syncwarp();
      const int4 ti = ts.d_info[tt];
      tag_tile<DIMS, TY, TZ, false>(ts.d_desc[ti.x], ti, tt, Q, seeds);
      ++visits;
    }
    ok = jfc::grid_sync(ctr, [&]() {
      ctr->ticket[cb] = 0;
      ctr->qn_bfs[cb] = 0;
    });
  }
  __shared__ unsigned long long s_vis;
  if (threadIdx.x == 0) s_vis = 0;
  __syncthreads();
  if (lane == 0 && visits) atomicAdd(&s_vis, visits);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (s_vis) atomicAdd(&ctr->bfs_visits, s_vis);
    if (blockIdx.x == 0) {
      ctr->bfs_passes = pass;
      if (ctr->bfs_status == 0) ctr->bfs_status = 1;
    }
  }
}

// ------------------------------------------------------------ global relabel
// x-direction closure of one tile row (lane = x): h(p) = min(h(p), h(q) + |p - q|)
// over the runs of residual arcs p -> p+1 -> ... -> q (axp) and p -> p-1 ->
// ... -> q (axm), by doubling.  The arc runs are read from the row's arc
// masks, so only the values move between lanes.
__device__ __forceinline__ int row_close(int v, unsigned axp, unsigned axm, int lane) {
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int nv = __shfl_down_sync(FULL, v, off);
    const unsigned run = (1u << off) - 1u;
    if (lane + off < 32 && ((~axp >> lane) & run) == 0u) v = min(v, nv + off);
  }
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int nv = __shfl_up_sync(FULL, v, off);
    const unsigned run = (1u << off) - 1u;
    if (lane >= off && ((~axm >> (lane - off + 1)) & run) == 0u) v = min(v, nv + off);
  }
  return v;
}

// In-tile closure of a warp's tile (lane = x, hv[i] = row i's height, lab[i]
// its arc byte, AXP / AXM the rows' x-arc masks): h(u) = min(h(u), h(v) + 1)
// over residual arcs u -> v inside the tile, to the fixpoint.  Row closures
// by doubling shuffles, y and z runs in registers (a backward and a forward
// sweep per line); bounded by the tile's nodes (every pass but the last
// lowers some height, and heights are bounded below by 0).  The row closures
// are what a visit costs (10 shuffles and 80 instructions a row), so only rows
// that something lowered since their last one get one, 4 at a time (their
// chains overlap); `rows`: the rows lowered before the call (the same in every
// lane).  With every row closed in every pass, and a last pass to see that
// nothing falls, the frontier took 48.2 ms of a 2560 x 1440 x 50 solve instead of
// 44.9.
template <int TY, int TZ>
__device__ __forceinline__ void tile_close(int (&hv)[TY * TZ], const unsigned (&lab)[TY * TZ],
                                           const unsigned (&AXP)[TY * TZ], const unsigned (&AXM)[TY * TZ], int lane,
                                           unsigned rows) {
  constexpr int R = TY * TZ;
  for (int pass = 0; rows != 0u && pass < 32 * R; ++pass) {
#pragma unroll
    for (int i0 = 0; i0 < R; i0 += 4) {
      if ((rows >> i0 & 15u) == 0u) continue;
#pragma unroll
      for (int i = i0; i < i0 + 4; ++i) hv[i] = row_close(hv[i], AXP[i], AXM[i], lane);
    }
    unsigned low = 0;   // rows lowered in this lane
    auto run = [&](int i, int from, unsigned arc) {
      if ((lab[i] & arc) && hv[from] + 1 < hv[i]) { hv[i] = hv[from] + 1; low |= 1u << i; }
    };
#pragma unroll
    for (int z = 0; z < TZ; ++z) {
#pragma unroll
      for (int y = TY - 2; y >= 0; --y) run(z * TY + y, z * TY + y + 1, jfc::A_YP);
#pragma unroll
      for (int y = 1; y < TY; ++y) run(z * TY + y, z * TY + y - 1, jfc::A_YM);
    }
#pragma unroll
    for (int y = 0; y < TY; ++y) {
#pragma unroll
      for (int z = TZ - 2; z >= 0; --z) run(z * TY + y, z * TY + y + TY, jfc::A_ZP);
#pragma unroll
      for (int z = 1; z < TZ; ++z) run(z * TY + y, z * TY + y - TY, jfc::A_ZM);
    }
    rows = __reduce_or_sync(FULL, low);
  }
}

// Row words of a 3D set, two uint4 per row segment of 32 nodes (bit = column):
// {+x, +y, +z, -z residual arcs}, {-y, -x residual arcs, deficit (e < 0), excess
// (e > 0)}; the cut keeps the reached nodes in the last word.
__device__ __forceinline__ uint4* row_words(const TileSet& ts, const GridDev& g, long long first, int y, int z, int c) {
  return ts.d_vf + 2 * (first + ((long long)z * g.Hp + y) * g.tiles_x + c);
}

// Row words and arc bytes of the tiles that something changed since the last
// relabel (28 bytes per node read; later passes read 1), one warp per tile; the
// counters of the relabel or cut that follows reset.
template <int TY, int TZ>
__global__ void __launch_bounds__(256, TY * TZ > 8 ? 1 : 2) k_bits3(TileSet ts) {
  constexpr int R = TY * TZ;
  using D = jfc::CtaTile<3, TY, TZ>;
  if (jfc::cycle_skips(ts)) return;
  DevCounters* ctr = ts.d_ctr;
  const int lane = threadIdx.x & 31;
  const long long gt = blockIdx.x * (long long)blockDim.x + threadIdx.x, gn = (long long)gridDim.x * blockDim.x;
  if (gt == 0) {
    ctr->t_gr_start = jfc::global_ns();
    jfc::begin_cycle(ts);
    ctr->bfs_status = 0;
    ctr->ticket[0] = ctr->ticket[1] = 0;
    ctr->qn_pr[0][0] = ctr->qn_pr[0][1] = ctr->qn_pr[1][0] = ctr->qn_pr[1][1] = 0;
    ctr->cur_pr[0] = ctr->cur_pr[1] = 0;
    ctr->wave_bar[0] = 0;
    ctr->q3_n[0] = ctr->q3_n[1] = ctr->q3_n[2] = 0;
    ctr->cut_bad = 0;
    ctr->pr_bar = 0;
  }
  for (long long i = gt; i < ts.ngrids; i += gn) {
    ts.d_grid_active[i] = 0;
    ts.d_grid_sum[2 * i] = ts.d_grid_sum[2 * i + 1] = 0;
  }
  for (long long t0 = gt - lane; t0 < ts.ntiles; t0 += gn) {
    unsigned todo = __ballot_sync(FULL, t0 + lane < ts.ntiles && ts.d_dirty[t0 + lane] != 0);
    while (todo) {
      const long long tid = t0 + __ffs(todo) - 1;
      todo &= todo - 1;
      const int4 ti = ts.d_info[tid];
      const GridDev& g = ts.d_desc[ti.x];
      const Addr a = make_addr<3, TY, TZ>(g, ti, lane);
      int e[R], r[6][R];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const long long n = roff<TY>(a, i);
        e[i] = g.e[n];
#pragma unroll
        for (int k = 0; k < 6; ++k) r[k][i] = g.r[k][n];
      }
      uint4 w0 = make_uint4(0, 0, 0, 0), w1 = w0;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        unsigned m[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) m[k] = __ballot_sync(FULL, r[k][i] > 0);
        const unsigned neg = __ballot_sync(FULL, e[i] < 0), pos = __ballot_sync(FULL, e[i] > 0);
        if (lane == i) {
          w0 = make_uint4(m[D::XP], m[D::YP], m[D::ZP], m[D::ZM]);
          w1 = make_uint4(m[D::YM], m[D::XM], neg, pos);
        }
        g.label[roff<TY>(a, i)] =
            (uint8_t)((r[D::XP][i] > 0 ? jfc::A_XP : 0u) | (r[D::YP][i] > 0 ? jfc::A_YP : 0u) |
                      (r[D::YM][i] > 0 ? jfc::A_YM : 0u) | (r[D::XM][i] > 0 ? jfc::A_XM : 0u) |
                      (r[D::ZP][i] > 0 ? jfc::A_ZP : 0u) | (r[D::ZM][i] > 0 ? jfc::A_ZM : 0u) |
                      (e[i] < 0 ? 64u : 0u) | (e[i] > 0 ? 128u : 0u));
      }
      if (lane < R) {
        uint4* w = row_words(ts, g, (long long)g.tile_base * R, a.y0 + lane % TY, a.z0 + lane / TY, ti.y);
        w[0] = w0;
        w[1] = w1;
      }
      if (lane == 0) ts.d_dirty[tid] = 0;
    }
  }
}

// First pass of the global relabel: in every tile a bit-parallel level BFS from
// its deficits (and from the deficits beside it), on the row words.  A lane
// holds one row, so a warp expands 32 / R tiles at once, a dozen word operations
// and four shuffles per level; 5 + 1 bits of level are kept per node and turned
// into heights 4 columns a lane.  A row of heights is written only where it
// differs from what the plane holds.  One byte of words and 4 bytes of heights
// read per node: with a warp per tile and every lane holding every row's words
// the pass took 2.2 ms on 2560 x 1440 x 50 (28 bytes read, 5 written per node,
// 32 times the same word operations), with k_bits3 it takes 0.48 (few tiles
// changed) to 0.78 ms (1.5 on a solve's first, which reads all planes).
template <int TY, int TZ>
__global__ void __launch_bounds__(256, 4) k_relabel_first(TileSet ts) {
  constexpr int R = TY * TZ, G = 32 / R, kPlanes = R > 8 ? 10 : 9;   // tiles a warp; bits of a level (at most 32 R)
  struct Row { unsigned v, def, p[kPlanes]; };
  __shared__ Row s_row[8][32];
  if (jfc::cycle_skips(ts)) return;
  DevCounters* ctr = ts.d_ctr;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int tid = (int)min(w * G + lane / R, (long long)ts.ntiles - 1);
  const bool ok = w * G + lane / R < ts.ntiles;
  if (w * G >= ts.ntiles) return;
  const int r = lane % R, y = r % TY, z = r / TY;
  const int4 ti = ts.d_info[tid];
  const GridDev& g = ts.d_desc[ti.x];
  const int gy = ti.z * TY + y, gz = ti.w * TZ + z;
  const long long first = (long long)g.tile_base * R;
  const bool xl = ti.y > 0, xr = ti.y + 1 < g.tiles_x, yt = gy > 0, yb = gy + 1 < g.Hp, zt = gz > 0, zb = gz + 1 < g.Dp;
  uint4 w0 = make_uint4(0, 0, 0, 0), w1 = w0;
  unsigned s1 = 0;   // nodes with a residual arc into a deficit outside the tile
  if (ok) {
    const uint4* rw = row_words(ts, g, first, gy, gz, ti.y);
    w0 = rw[0];
    w1 = rw[1];
    auto neg = [&](int dy, int dz, int dc) { return row_words(ts, g, first, gy + dy, gz + dz, ti.y + dc)[1].z; };
    if (xl) s1 |= neg(0, 0, -1) >> 31 & w1.y;
    if (xr) s1 |= neg(0, 0, 1) << 31 & w0.x;
    if (y == 0 && yt) s1 |= neg(-1, 0, 0) & w1.x;
    if (y == TY - 1 && yb) s1 |= neg(1, 0, 0) & w0.y;
    if (z == 0 && zt) s1 |= neg(0, -1, 0) & w0.w;
    if (z == TZ - 1 && zb) s1 |= neg(0, 1, 0) & w0.z;
  }
  const unsigned def = w1.z, pos = w1.w;
  unsigned V = def, F = def, P[kPlanes];
#pragma unroll
  for (int b = 0; b < kPlanes; ++b) P[b] = 0;
  const int dmax = jfc::cap_of(g, ctr) - 1;   // (levels at or above the cap stay unreachable)
  int d = 1;
  for (; d <= 32 * R; ++d) {
    const unsigned up = __shfl_up_sync(FULL, F, 1), dn = __shfl_down_sync(FULL, F, 1);
    unsigned m = (F >> 1 & w0.x) | (F << 1 & w1.y);
    if (y > 0) m |= up & w1.x;
    if (y < TY - 1) m |= dn & w0.y;
    if constexpr (TZ > 1) {
      const unsigned fr = __shfl_down_sync(FULL, F, TY), bk = __shfl_up_sync(FULL, F, TY);
      if (z < TZ - 1) m |= fr & w0.z;
      if (z > 0) m |= bk & w0.w;
    }
    if (d == 1) m |= s1;
    const unsigned N = d <= dmax ? m & ~V : 0u;
    if (!__any_sync(FULL, N != 0u)) break;
    V |= N;
    F = N;
#pragma unroll
    for (int b = 0; b < kPlanes; ++b)
      if (d >> b & 1) P[b] |= N;
  }
  const int bits = 32 - __clz(d);   // of the levels that occur
  Row& o = s_row[warp][lane];
  o.v = V;
  o.def = def;
#pragma unroll
  for (int b = 0; b < kPlanes; ++b) o.p[b] = P[b];
  int* const hrow = ok ? g.h + (long long)ti.y * 32 + (long long)gy * g.pitch + (long long)gz * g.pitch * g.Hp : nullptr;
  __syncwarp();
#pragma unroll 2
  for (int k = 0; k < 8; ++k) {
    const int row = 4 * k + (lane >> 3), sh = 4 * (lane & 7);
    int* h = reinterpret_cast<int*>(__shfl_sync(FULL, (unsigned long long)hrow, row));
    const Row& q = s_row[warp][row];
    if (!h) continue;
    const int4 old = *reinterpret_cast<const int4*>(h + sh);
    const unsigned vn = q.v >> sh & 15u, dn = q.def >> sh & 15u;
    unsigned lo = 0, hi = 0;   // the 4 columns' levels, a byte each
#pragma unroll
    for (int b = 0; b < 8; ++b)
      if (b < bits) lo |= (((q.p[b] >> sh & 15u) * 0x00204081u) & 0x01010101u) << b;
    if (bits > 8) {
#pragma unroll
      for (int b = 8; b < kPlanes; ++b) hi |= (((q.p[b] >> sh & 15u) * 0x00204081u) & 0x01010101u) << (b - 8);
    }
    auto val = [&](int c) -> int {
      const int l = (int)(lo >> (8 * c) & 255u) | (int)(hi >> (8 * c) & 255u) << 8;
      return dn >> c & 1u ? 0 : vn >> c & 1u ? l : JFC_INF;
    };
    const int4 nw = make_int4(val(0), val(1), val(2), val(3));
    if (nw.x != old.x || nw.y != old.y || nw.z != old.z || nw.w != old.w) *reinterpret_cast<int4*>(h + sh) = nw;
  }
  // ---- activity, and the neighbours whose halo holds news (finite and above 0)
  const unsigned group = (R == 32 ? FULL : (1u << R) - 1u) << (lane / R * R);
  const unsigned fin = ok ? V & ~def : 0u;
  const bool act = (__ballot_sync(FULL, ok && (pos & V) != 0u) & group) != 0u;
  const unsigned bx0 = __ballot_sync(FULL, (fin & 1u) != 0u), bx1 = __ballot_sync(FULL, fin >> 31 != 0u);
  const unsigned by0 = __ballot_sync(FULL, y == 0 && fin), by1 = __ballot_sync(FULL, y == TY - 1 && fin);
  const unsigned bz0 = __ballot_sync(FULL, z == 0 && fin), bz1 = __ballot_sync(FULL, z == TZ - 1 && fin);
  const int txs = g.tiles_x, txy = g.tiles_x * g.tiles_y;
  bool want = false;
  int nb = tid;
  switch (ok ? r : 7) {
    case 0: want = (bx0 & group) && xl; nb = tid - 1; break;
    case 1: want = (bx1 & group) && xr; nb = tid + 1; break;
    case 2: want = (by0 & group) && ti.z > 0; nb = tid - txs; break;
    case 3: want = (by1 & group) && ti.z + 1 < g.tiles_y; nb = tid + txs; break;
    case 4: want = (bz0 & group) && ti.w > 0; nb = tid - txy; break;
    case 5: want = (bz1 & group) && ti.w + 1 < g.tiles_z; nb = tid + txy; break;
    default: break;
  }
  jfc::warp_append(want, nb, ts.d_flag_bfs[1], ts.d_q_bfs[1], &ctr->q3_n[1]);
  if (ok && r == 0) ts.d_act[tid] = act ? 1 : 0;
  const unsigned lead = __ballot_sync(FULL, ok && r == 0 && act);
  if (ts.ngrids == 1) {
    if (lane == 0 && lead) atomicAdd(&ts.d_grid_active[0], __popc(lead));
  } else if (ok && r == 0 && act) {
    atomicAdd(&ts.d_grid_active[ti.x], 1);
  }
}

// Frontier visit, one warp per tile, min-plus form: the tile's heights in
// registers (lane = x, one register per row), lowered by the halo heights
// across residual arcs, then closed in place: row closures by doubling
// shuffles, y and z runs in registers (a forward and a backward sweep per
// line), repeated until nothing falls.  Monotone, so the fixpoint is the
// exact in-tile distance given the halo, as the level BFS gives; a visit
// costs one closure per turn a shortest path takes instead of one step per
// level.  Improvements at or above the distance cap are dropped (those
// nodes stay unreachable).
// Staged tile of a 3D frontier visit, filled by two tensor copies: the h
// plane over the tile and its one-cell halo (40 columns from x0 - 4, as the
// push-relabel staging) and the tile's arc bytes.
template <int TY, int TZ>
struct alignas(128) RlStage {
  using T = jfc::CtaTile<3, TY, TZ, 40, 4>;
  static constexpr unsigned kHb = sizeof(int) * T::HN, kLb = 32u * TY * TZ;
  static constexpr unsigned kBytes = kHb + kLb;   // bytes the two copies deliver
  int hb[T::HN];
  alignas(128) uint8_t lb[32 * TY * TZ];
};

// hb / lb non-null: the tile comes from a staged copy (RlStage) instead of
// global loads.
template <int TY, int TZ, bool STAGED = false>
__device__ __forceinline__ void relabel_frontier_minplus(const TileSet& ts, int tid, int4 ti, const BfsQ& Q,
                                                         int& cur_grid, int& delta, const int* hb = nullptr,
                                                         const uint8_t* lb = nullptr) {
  constexpr int R = TY * TZ;
  using ST = jfc::CtaTile<3, TY, TZ, 40, 4>;
  const int lane = threadIdx.x & 31;
  const GridDev& g = ts.d_desc[ti.x];
  const Addr a = make_addr<3, TY, TZ>(g, ti, lane);
  // the tile's activity byte as the last visit left it (another SM's write of
  // an earlier pass: read from L2, and early, so its latency overlaps the
  // closure)
  const unsigned act_old = lane == 0 ? (unsigned)__ldcg(ts.d_act + tid) : 0u;
  unsigned lab[R];
  int hv[R], h0[R];
  unsigned AXP[R], AXM[R];
  unsigned posm = 0;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    if constexpr (STAGED) {
      lab[i] = lb[i * 32 + lane];
      h0[i] = hb[ST::hidx(lane, i % TY, i / TY)];
    } else {
      const long long n = roff<TY>(a, i);
      lab[i] = g.label[n];   // arc byte written by the first pass
      h0[i] = g.h[n];
    }
  }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    hv[i] = h0[i];
    AXP[i] = __ballot_sync(FULL, lab[i] & jfc::A_XP);
    AXM[i] = __ballot_sync(FULL, lab[i] & jfc::A_XM);
    if (lab[i] & 128u) posm |= 1u << i;
  }
  // the halo, fixed during the visit: y faces per z slice (lane = x), z
  // faces per row y, x faces in lanes r (left of row r) and 16 + r (right);
  // loaded together with the tile (no load waits for the arc bytes)
  int HT[TZ], HB[TZ], HZT[TY], HZB[TY];
#pragma unroll
  for (int z = 0; z < TZ; ++z) {
    if constexpr (STAGED) {
      HT[z] = a.has_yT ? hb[ST::hidx(lane, -1, z)] : JFC_INF;
      HB[z] = a.has_yB ? hb[ST::hidx(lane, TY, z)] : JFC_INF;
    } else {
      const long long n = roff<TY>(a, z * TY);
      HT[z] = a.has_yT ? g.h[n - a.pitch] : JFC_INF;
      HB[z] = a.has_yB ? g.h[n + (long long)TY * a.pitch] : JFC_INF;
    }
  }
#pragma unroll
  for (int y = 0; y < TY; ++y) {
    if constexpr (STAGED) {
      HZT[y] = a.has_zT ? hb[ST::hidx(lane, y, -1)] : JFC_INF;
      HZB[y] = a.has_zB ? hb[ST::hidx(lane, y, TZ)] : JFC_INF;
    } else {
      const long long n = roff<TY>(a, y);
      HZT[y] = a.has_zT ? g.h[n - a.slab] : JFC_INF;
      HZB[y] = a.has_zB ? g.h[n + (long long)TZ * a.slab] : JFC_INF;
    }
  }
  const int xrow = lane & 15;
  int hx = JFC_INF;
  if (xrow < R && (lane < 16 ? a.has_xL : a.has_xR))
    hx = STAGED ? hb[ST::hidx(lane < 16 ? -1 : 32, xrow % TY, xrow / TY)]
                : g.h[(long long)(lane < 16 ? a.x0 - 1 : a.x0 + 32) + (long long)(a.y0 + xrow % TY) * a.pitch +
                  (long long)(a.z0 + xrow / TY) * a.slab];
  // the tile's interior is at its fixpoint (the dense pass or its last
  // visit closed it, and only its own visits write it), so only a halo seed
  // that lowers a border node can change anything
  unsigned seeded = 0;   // rows lowered by the halo in this lane
  auto seed = [&](int i, bool arc, int hn) {
    if (arc && hn + 1 < hv[i]) { hv[i] = hn + 1; seeded |= 1u << i; }
  };
#pragma unroll
  for (int z = 0; z < TZ; ++z) {
    const int it = z * TY, ib = z * TY + TY - 1;
    seed(it, lab[it] & jfc::A_YM, HT[z]);
    seed(ib, lab[ib] & jfc::A_YP, HB[z]);
  }
#pragma unroll
  for (int y = 0; y < TY; ++y) {
    const int it = y, ib = (TZ - 1) * TY + y;
    seed(it, lab[it] & jfc::A_ZM, HZT[y]);
    seed(ib, lab[ib] & jfc::A_ZP, HZB[y]);
  }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int hl = __shfl_sync(FULL, hx, i), hr = __shfl_sync(FULL, hx, 16 + i);
    seed(i, lane == 0 && (lab[i] & jfc::A_XM), hl);
    seed(i, lane == 31 && (lab[i] & jfc::A_XP), hr);
  }
  tile_close<TY, TZ>(hv, lab, AXP, AXM, lane, __reduce_or_sync(FULL, seeded));
  const int cap = jfc::cap_of(g, ts.d_ctr);
  unsigned rows_changed = 0;
  bool c0 = false, c31 = false, act = false;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    if (hv[i] >= cap) hv[i] = h0[i];   // at or above the cap: stays as it was (unreachable)
    const bool chg = hv[i] < h0[i];
    const unsigned m = __ballot_sync(FULL, chg);
    if (m) {
      rows_changed |= 1u << i;
      c0 |= (m & 1u) != 0;
      c31 |= (m >> 31) != 0;
    }
    if (chg) g.h[roff<TY>(a, i)] = hv[i];
    act |= ((posm >> i) & 1u) && hv[i] < JFC_INF;
  }
  act = __any_sync(FULL, act);
  if (lane == 0) {
    const int old = act_old != 0 ? 1 : 0;
    ts.d_act[tid] = act ? 1 : 0;
    if (ti.x != cur_grid) {
      if (delta && cur_grid >= 0) atomicAdd(&ts.d_grid_active[cur_grid], delta);
      delta = 0;
      cur_grid = ti.x;
    }
    delta += (act ? 1 : 0) - old;
  }
  flag_neighbours<3, TY, TZ>(g, a, tid, rows_changed, c0, c31, false, Q);
}

// Refill of the push-relabel queues (buffer 0 of each parity) from the
// active-tile flags, warp-aggregated.
__device__ __forceinline__ void refill_pr_queues(const TileSet& ts, DevCounters* ctr, int warp, int nwarps, int lane) {
  for (long long b = 32ll * warp; b < ts.ntiles; b += 32ll * nwarps) {
    const long long t = b + lane;
    const bool act = t < ts.ntiles && __ldcg(ts.d_act + t) != 0;
    int par = 0;
    if (act) { const int4 ti = ts.d_info[t]; par = (ti.y + ti.z + ti.w) & 1; }
    if (t < ts.ntiles) ts.d_flag_pr[t] = act ? 1 : 0;
    jfc::warp_append(act && par == 0, (int)t, nullptr, ts.d_q_pr[0][0], &ctr->qn_pr[0][0]);
    jfc::warp_append(act && par == 1, (int)t, nullptr, ts.d_q_pr[1][0], &ctr->qn_pr[1][0]);
  }
}

// Global relabel, frontier passes (persistent, cooperative): one warp per queued
// tile, a grid barrier between passes, until a pass queues nothing; then the
// push-relabel queues are refilled with every tile holding an active node (the
// reference's graphcut_count_node + clogs scan + graphcut_scatter_node,
// graphcut_count_block.cl:19-65, as one warp-aggregated append).
// A pass holds a few tiles per warp and its time is a chain of latencies, so
// every nwarps-th queue entry is a warp's own, consecutive ones on different
// SMs: a warp reads up to 32 entries and their tiles at once.  (By tickets, with
// the next two tiles' tickets, entries and coordinates fetched one after the
// other before each visit, and barriers of 3 us, the frontier took
// 27.2 ms of a 2560 x 1440 x 50 solve instead of 23.5, 3.25 of a 640 x 400 x 20 one
// instead of 2.38.)
// (2 CTAs per SM, the registers the staging holds without spills: 3 CTAs per
// SM spilled and measured slower, 116.5 vs 104-108.5 ms of frontier per video
// solve)
#ifndef JFC_RL3D_MINB
#define JFC_RL3D_MINB 2
#endif
// 1: 3D frontier tiles of up to 8 rows are staged by tensor copies
#ifndef JFC_RL3D_STAGE
#define JFC_RL3D_STAGE 1
#endif
template <int TY, int TZ>
__global__ void __launch_bounds__(256, TY * TZ > 8 ? 2 : JFC_RL3D_MINB)
    k_relabel_warp(TileSet ts, int max_passes) {
  if (jfc::cycle_skips(ts)) return;
  __shared__ int s_items[8][64];   // per-warp staged queue appends (at most 38 before a flush)
  __shared__ int s_cnt[8];
  // 3D tiles of up to 8 rows with tensor maps: each warp stages its tiles by
  // tensor copies into two buffers of its own (dynamic shared memory), the
  // next entry's tile copied while the current one is visited
  using Stage = RlStage<TY, TZ>;
  constexpr bool kStage = JFC_RL3D_STAGE && TY * TZ <= 8;
  __shared__ uint64_t s_bar[8][2];
  extern __shared__ __align__(128) unsigned char s_dyn[];
  DevCounters* ctr = ts.d_ctr;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gw = warp * (int)gridDim.x + (int)blockIdx.x, nw = (int)(gridDim.x * (blockDim.x >> 5));
  const bool tma = kStage && ts.d_tmap != nullptr;
  Stage* stage = reinterpret_cast<Stage*>(s_dyn + ((128u - (jfc::smem_addr(s_dyn) & 127u)) & 127u)) + 2 * warp;
  if (lane == 0) s_cnt[warp] = 0;
  if (tma && lane == 0) {
    jfc::mbar_init(&s_bar[warp][0], 1);
    jfc::mbar_init(&s_bar[warp][1], 1);
    jfc::fence_mbar_init();
  }
  __syncthreads();
  const unsigned long long spin = jfc::spin_cap(ctr);
  unsigned parity = 0;      // bit b: phase parity of buffer b's next fill (warp-uniform)
  int acquired_grid = -1;   // lane 0: grid whose maps it acquired
  // lane 0: copy tile t4 (grid, tile x / y / z) into buffer b
  auto issue = [&](int4 t4, int b) {
    if (lane == 0) {
      const char* maps = (const char*)ts.d_tmap + (size_t)t4.x * 384;
      if (t4.x != acquired_grid) {
        jfc::fence_tmap_acquire(maps + 128);
        jfc::fence_tmap_acquire(maps + 256);
        acquired_grid = t4.x;
      }
      jfc::fence_async_shared();
      jfc::mbar_arrive_tx(&s_bar[warp][b], Stage::kBytes);
      jfc::tma_load_3d(stage[b].hb, maps + 128, t4.y * 32 - 4, t4.z * TY - 1, t4.w * TZ - 1, &s_bar[warp][b]);
      jfc::tma_load_3d(stage[b].lb, maps + 256, t4.y * 32, t4.z * TY, t4.w * TZ, &s_bar[warp][b]);
    }
  };
  unsigned long long visits = 0;
  int cur_grid = -1, delta = 0;
  bool ok = true;
  int pass = 1;
  const unsigned long long t1 = jfc::global_ns();
  for (pass = 1; ok; ++pass) {
    const int cb = pass & 1;
    const int n = jfc::vload(&ctr->q3_n[pass % 3]);
    if (n == 0) break;
    if (pass > max_passes) {
      if (blockIdx.x == 0 && threadIdx.x == 0) ctr->bfs_status = 2;
      break;
    }
    BfsQ Q{ts.d_flag_bfs[cb ^ 1], ts.d_q_bfs[cb ^ 1], &ctr->q3_n[(pass + 1) % 3], s_items[warp], &s_cnt[warp]};
    const int* queue = ts.d_q_bfs[cb];
    int* fcur = ts.d_flag_bfs[cb];
    // (every CTA has read the count of the pass before; it is the one after next's)
    if (blockIdx.x == 0 && threadIdx.x == 0) ctr->q3_n[(pass + 2) % 3] = 0;
    // the previous pass's writes (seen through the grid barrier) come before
    // this pass's tensor reads
    if (tma && lane == 0) jfc::fence_async_global();
    const int mine = n > gw ? (n - gw + nw - 1) / nw : 0;   // entries gw, gw + nw, ...
    bool got = true;
    for (int b = 0; b < mine && got; b += 32) {
      const int cnt = min(32, mine - b);
      const int my_t = lane < cnt ? __ldcg(queue + gw + (b + lane) * nw) : 0;
      const int4 my_ti = lane < cnt ? ts.d_info[my_t] : make_int4(0, 0, 0, 0);
      if (lane < cnt) fcur[my_t] = 0;
      auto tile = [&](int j) {
        return make_int4(__shfl_sync(FULL, my_ti.x, j), __shfl_sync(FULL, my_ti.y, j), __shfl_sync(FULL, my_ti.z, j),
                         __shfl_sync(FULL, my_ti.w, j));
      };
      // entry j is staged in buffer j & 1, the next one being copied into the other
      if (tma) {
        issue(tile(0), 0);
        if (cnt > 1) issue(tile(1), 1);
      }
      for (int j = 0; j < cnt; ++j) {
        const int tt = __shfl_sync(FULL, my_t, j), buf = j & 1;
        const int4 ti = tile(j);
        __syncwarp();
        if (tma) {
          const unsigned ph = (parity >> buf) & 1u;
          got = __all_sync(FULL, jfc::mbar_wait(&s_bar[warp][buf], ph, spin));
          parity ^= 1u << buf;
          if (!got) {
            if (lane == 0) {
              atomicExch(&ctr->error, 1);
              // copies in flight land before the warp leaves (fixed bound)
              constexpr unsigned long long kDrainPolls = 1ull << 26;
              jfc::mbar_wait(&s_bar[warp][buf], ph, kDrainPolls);
              if (j + 1 < cnt) jfc::mbar_wait(&s_bar[warp][buf ^ 1], (parity >> (buf ^ 1)) & 1u, kDrainPolls);
            }
            __syncwarp();
            break;   // the grid barrier below sees the error: every CTA leaves
          }
          relabel_frontier_minplus<TY, TZ, true>(ts, tt, ti, Q, cur_grid, delta, stage[buf].hb, stage[buf].lb);
          __syncwarp();   // every lane has read `buf` before it is refilled
          if (j + 2 < cnt) issue(tile(j + 2), buf);
        } else {
          relabel_frontier_minplus<TY, TZ>(ts, tt, ti, Q, cur_grid, delta);
        }
        ++visits;
        __syncwarp();
        if (*(volatile int*)Q.scnt >= 32) {
          flush_staged(Q, lane);
          __syncwarp();
          if (lane == 0) *Q.scnt = 0;
          __syncwarp();
        }
      }
    }
    __syncwarp();
    flush_staged(Q, lane);
    __syncwarp();
    if (lane == 0) *Q.scnt = 0;
    __syncwarp();
    ok = jfc::arrive_wait(ctr, ctr->wave_bar, (unsigned long long)pass * gridDim.x);
  }
  if (lane == 0 && delta && cur_grid >= 0) atomicAdd(&ts.d_grid_active[cur_grid], delta);
  if (ok) refill_pr_queues(ts, ctr, gw, nw, lane);
  // frontier visits are counted per warp (lane 0); pass 0 visited every tile
  __shared__ unsigned long long s_vis;
  if (threadIdx.x == 0) s_vis = 0;
  __syncthreads();
  if (lane == 0 && visits) atomicAdd(&s_vis, visits);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (s_vis) atomicAdd(&ctr->bfs_visits, s_vis);
    if (blockIdx.x == 0) {
      ctr->bfs_passes = pass;
      ctr->bfs_visits += (unsigned long long)ts.ntiles;
      if (ctr->bfs_status == 0) ctr->bfs_status = 1;
      const unsigned long long t2 = jfc::global_ns();
      ctr->ns_gr_first += t1 - ctr->t_gr_start;
      ctr->ns_gr_frontier += t2 - t1;
    }
  }
}

// Cut of a 3D set (graphcut_init_cut / graphcut_compute_cut,
// graphcut_compute_cut.cl:74-140): the source side is every node reachable from
// {e > 0} along residual arcs; reaching a deficit raises cut_bad (the
// reference's done[1] divergence flag).  On the row words: a warp holds a block
// of BY x BZ = 32 rows (whole tiles, named by the first of them), a lane one
// row, so a step closes all rows with a dozen word operations and exchanges the
// reached nodes with four shuffles.  The reached nodes stay in the rows' last
// word; only the block's warp writes them and they only grow, so the blocks
// around may read them at any time.  The first pass visits every block; a block
// whose border an arc from a newly reached node to an unreached one crosses
// queues the block behind it for the next pass; a last pass writes the label
// bytes and sums min(e, 0) and the labels per grid.  What bounds it is the
// first pass's bytes (1 read per node, 5 in the last) and then the chain of
// passes.  A pass of a warp per 8-row tile with every row's words in every
// lane, from e and the arcs (29 bytes per node), and the separate sums took 0.45
// ms on 317 x 301 x 181 and 4.2 ms on 2560 x 1440 x 50; this takes 0.12 and 0.77
// (0.20 of it the excess and label planes at the HBM rate).
template <int TY, int TZ>
__global__ void __launch_bounds__(256, 4) k_cut3(TileSet ts, int max_passes) {
  constexpr int BY = TY > 8 ? TY : 8, BZ = 32 / BY, MY = BY / TY, MZ = BZ / TZ;
  constexpr int kList = 1024, kScan = 8;   // staged appends of a CTA; tiles a warp looks through at once
  __shared__ int s_list[kList];
  __shared__ int s_n, s_base;
  __shared__ unsigned long long s_sum[2], s_vis;
  if (jfc::cycle_skips(ts)) return;
  DevCounters* ctr = ts.d_ctr;
  const int t = threadIdx.x, lane = t & 31;
  const int warp = (int)((blockIdx.x * blockDim.x + t) >> 5), nwarps = (int)(gridDim.x * blockDim.x >> 5);
  if (t == 0) {
    s_n = 0;
    s_sum[0] = s_sum[1] = s_vis = 0;
  }
  __syncthreads();
  struct Row { int y, z; bool ok; uint4* w; };
  auto row_of = [&](const GridDev& g, int4 ti, int r) {
    Row q;
    q.y = ti.z * TY + r % BY;
    q.z = ti.w * TZ + r / BY;
    q.ok = q.y < g.Hp && q.z < g.Dp;
    q.w = row_words(ts, g, (long long)g.tile_base * (TY * TZ), q.y, q.z, ti.y);
    return q;
  };
  // f(tile, info) for every block of this warp
  auto each_block = [&](auto f) {
    for (long long t0 = (long long)warp * kScan; t0 < ts.ntiles; t0 += (long long)nwarps * kScan) {
      const bool in = lane < kScan && t0 + lane < ts.ntiles;
      const int4 mine = in ? ts.d_info[t0 + lane] : make_int4(0, 0, 0, 0);
      unsigned todo = __ballot_sync(FULL, in && mine.z % MY == 0 && mine.w % MZ == 0);
      while (todo) {
        const int k = __ffs(todo) - 1;
        todo &= todo - 1;
        f((int)t0 + k, make_int4(__shfl_sync(FULL, mine.x, k), __shfl_sync(FULL, mine.y, k),
                                 __shfl_sync(FULL, mine.z, k), __shfl_sync(FULL, mine.w, k)));
      }
    }
  };
  unsigned visits = 0;
  int pass = 0;
  auto visit = [&](int tid, int4 ti) {
    const GridDev& g = ts.d_desc[ti.x];
    const Row q = row_of(g, ti, lane);
    const int y = lane % BY, z = lane / BY;
    const long long sy = 2ll * g.tiles_x, sz = sy * g.Hp;   // words to the next row, slice
    uint4 w0 = make_uint4(0, 0, 0, 0), w1 = w0;
    // words beside the row, and their arcs toward it; what lies behind the block's border
    unsigned lw = ~0u, rw = ~0u, yw = ~0u, zw = ~0u, la = 0, ra = 0, ya = 0, za = 0;
    if (q.ok) {
      w0 = q.w[0];
      w1 = __ldcg(q.w + 1);
      if (ti.y > 0) { lw = __ldcg(&q.w[-1].w); la = q.w[-2].x; }
      if (ti.y + 1 < g.tiles_x) { rw = __ldcg(&q.w[3].w); ra = q.w[3].y; }
      if (y == 0 && q.y > 0) { yw = __ldcg(&q.w[1 - sy].w); ya = q.w[-sy].y; }
      if (y == BY - 1 && q.y + 1 < g.Hp) { yw = __ldcg(&q.w[1 + sy].w); ya = q.w[1 + sy].x; }
      if (z == 0 && q.z > 0) { zw = __ldcg(&q.w[1 - sz].w); za = q.w[-sz].z; }
      if (z == BZ - 1 && q.z + 1 < g.Dp) { zw = __ldcg(&q.w[1 + sz].w); za = q.w[sz].w; }
    }
    const unsigned L0 = w1.w;
    unsigned L = L0 | (lw & la) >> 31 | (rw & ra) << 31 | (yw & ya) | (zw & za);
    for (int it = 0; it < 32 * 32; ++it) {   // (a step but the last reaches a node)
      const unsigned was = L;
      L = jfc::close_left(jfc::close_right(L, w0.x << 1), w1.y >> 1);
      const unsigned up = __shfl_up_sync(FULL, L & w0.y, 1), dn = __shfl_down_sync(FULL, L & w1.x, 1);
      const unsigned fr = __shfl_up_sync(FULL, L & w0.z, BY), bk = __shfl_down_sync(FULL, L & w0.w, BY);
      if (y > 0) L |= up;
      if (y < BY - 1) L |= dn;
      if (z > 0) L |= fr;
      if (z < BZ - 1) L |= bk;
      if (!__any_sync(FULL, L != was)) break;
    }
    const unsigned news = L & ~L0;
    if (news) q.w[1].w = L;
    if (L & w1.z) ctr->cut_bad = 1;
    unsigned dirs = (news & w1.y & 1u & ~(lw >> 31)) | ((news & w0.x) >> 31 & ~rw) << 1;
    if (y == 0 && (news & w1.x & ~yw)) dirs |= 4u;
    if (y == BY - 1 && (news & w0.y & ~yw)) dirs |= 8u;
    if (z == 0 && (news & w0.w & ~zw)) dirs |= 16u;
    if (z == BZ - 1 && (news & w0.z & ~zw)) dirs |= 32u;
    dirs = __reduce_or_sync(FULL, dirs);
    if (lane < 6 && (dirs >> lane & 1u)) {
      const int step = lane < 2 ? 1 : lane < 4 ? MY * g.tiles_x : MZ * g.tiles_x * g.tiles_y;
      const int nb = lane & 1 ? tid + step : tid - step, b = (pass + 1) & 1;
      if (atomicExch(ts.d_flag_bfs[b] + nb, 1) == 0) {
        const int i = atomicAdd(&s_n, 1);
        if (i < kList) s_list[i] = nb;
        else ts.d_q_bfs[b][atomicAdd(&ctr->q3_n[(pass + 1) % 3], 1)] = nb;
      }
    }
    ++visits;
  };
  bool ok = true;
  for (;; ++pass) {
    if (pass == 0) {
      each_block(visit);
    } else {
      const int n = jfc::vload(&ctr->q3_n[pass % 3]);
      if (n == 0) break;
      if (pass > max_passes) {
        if (blockIdx.x == 0 && t == 0) ctr->bfs_status = 2;
        ok = false;
        break;
      }
      for (int k = warp; k < n; k += nwarps) {
        const int tid = __ldcg(ts.d_q_bfs[pass & 1] + k);
        if (lane == 0) ts.d_flag_bfs[pass & 1][tid] = 0;
        visit(tid, ts.d_info[tid]);
      }
      // (every CTA has read the count of the pass before; it is the one after next's)
      if (blockIdx.x == 0 && t == 0) ctr->q3_n[(pass + 2) % 3] = 0;
    }
    __syncthreads();
    const int staged = min(s_n, kList);
    if (staged) {
      if (t == 0) s_base = atomicAdd(&ctr->q3_n[(pass + 1) % 3], staged);
      __syncthreads();
      for (int i = t; i < staged; i += blockDim.x) ts.d_q_bfs[(pass + 1) & 1][s_base + i] = s_list[i];
      __syncthreads();
      if (t == 0) s_n = 0;
    }
    ok = jfc::arrive_wait(ctr, &ctr->pr_bar, (unsigned long long)(pass + 1) * gridDim.x);
    if (!ok) break;
  }
  // ---- labels (4 nodes a lane) and sums
  if (ok) {
    long long neg = 0, lab = 0;
    int cur = 0;
    auto add = [&]() {
      for (int o = 16; o; o >>= 1) {
        neg += __shfl_xor_sync(FULL, neg, o);
        lab += __shfl_xor_sync(FULL, lab, o);
      }
      if (lane == 0 && (neg || lab)) {
        unsigned long long* sum = ts.ngrids == 1 ? s_sum : (unsigned long long*)ts.d_grid_sum + 2 * cur;
        atomicAdd(sum, (unsigned long long)neg);
        atomicAdd(sum + 1, (unsigned long long)lab);
      }
      neg = lab = 0;
    };
    each_block([&](int, int4 ti) {
      if (ti.x != cur) {
        add();
        cur = ti.x;
      }
      const GridDev& g = ts.d_desc[ti.x];
      const Row q = row_of(g, ti, lane);
      const unsigned L = q.ok ? __ldcg(&q.w[1].w) : 0u;
      lab += __popc(L);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int r = 4 * k + (lane >> 3), sh = 4 * (lane & 7);
        const unsigned nib = __shfl_sync(FULL, L, r) >> sh & 15u;
        const int ry = ti.z * TY + r % BY, rz = ti.w * TZ + r / BY;
        if (ry >= g.Hp || rz >= g.Dp) continue;
        const long long n = (long long)ti.y * 32 + sh + (long long)g.pitch * (ry + (long long)g.Hp * rz);
        const int4 e = *reinterpret_cast<const int4*>(g.e + n);
        *reinterpret_cast<unsigned*>(g.label + n) = (nib * 0x00204081u) & 0x01010101u;
        neg += (long long)min(e.x, 0) + min(e.y, 0) + min(e.z, 0) + min(e.w, 0);
      }
    });
    add();
  }
  if (lane == 0) atomicAdd(&s_vis, (unsigned long long)visits * (MY * MZ));
  __syncthreads();
  if (t == 0) {
    if (ok && ts.ngrids == 1) {
      atomicAdd((unsigned long long*)ts.d_grid_sum, s_sum[0]);
      atomicAdd((unsigned long long*)ts.d_grid_sum + 1, s_sum[1]);
    }
    atomicAdd(&ctr->bfs_visits, s_vis);
    if (blockIdx.x == 0) {
      ctr->bfs_passes = pass;
      ctr->ns_cut = jfc::global_ns() - ctr->t_gr_start;
      if (ok) ctr->bfs_status = 1;
    }
  }
}

// (a launch of its own: in k_relabel_warp it changed the visits' registers and made
// the frontier 15% slower)
__global__ void k_end_cycle(TileSet ts) {
  if (!jfc::cycle_skips(ts)) jfc::end_cycle(ts);
}

// per-grid sum of min(e, 0) and count of source-side nodes (reduce_flow,
// bin/x64/cl/Infrastructures/reduce.cl:92-117, in int64 instead of int32 partials)
template <int TY, int TZ>
__global__ void __launch_bounds__(256) k_grid_sums(const GridDev* __restrict__ gd,
                                                   const int4* __restrict__ info, int ntiles,
                                                   long long* __restrict__ sums) {
  constexpr int R = TY * TZ;
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  int cur = -1;
  long long s_neg = 0, s_lab = 0;
  for (int t = warp; t < ntiles; t += nwarps) {
    const int4 ti = info[t];
    if (ti.x != cur) {
      if (cur >= 0) {
        for (int o = 16; o; o >>= 1) { s_neg += __shfl_xor_sync(FULL, s_neg, o); s_lab += __shfl_xor_sync(FULL, s_lab, o); }
        if (lane == 0) { atomicAdd((unsigned long long*)&sums[2 * cur], (unsigned long long)s_neg);
                         atomicAdd((unsigned long long*)&sums[2 * cur + 1], (unsigned long long)s_lab); }
      }
      s_neg = 0; s_lab = 0; cur = ti.x;
    }
    const GridDev& g = gd[ti.x];
    const long long pitch = g.pitch, slab = (long long)g.pitch * g.Hp;
    const long long base = (long long)(ti.y * 32 + lane) + (long long)ti.z * TY * pitch + (long long)ti.w * TZ * slab;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const long long n = base + (long long)(i % TY) * pitch + (long long)(i / TY) * slab;
      const int e = g.e[n];
      s_neg += e < 0 ? e : 0;
      s_lab += g.label[n];
    }
  }
  if (cur >= 0) {
    for (int o = 16; o; o >>= 1) { s_neg += __shfl_xor_sync(FULL, s_neg, o); s_lab += __shfl_xor_sync(FULL, s_lab, o); }
    if (lane == 0) { atomicAdd((unsigned long long*)&sums[2 * cur], (unsigned long long)s_neg);
                     atomicAdd((unsigned long long*)&sums[2 * cur + 1], (unsigned long long)s_lab); }
  }
}

// MODE 0: global relabel, 1: cut, 2: tag
template <int DIMS, int TY, int TZ, int MODE>
cudaError_t bfs_t(const TileSet& ts, int max_passes, const uint8_t* seeds, cudaStream_t s) {
  const void* fn;
  if constexpr (MODE == 1) fn = (const void*)k_cut3<TY, TZ>;
  else if constexpr (MODE == 2) fn = (const void*)k_tag<DIMS, TY, TZ>;
  else fn = (const void*)k_relabel_warp<TY, TZ>;
  const int nt = 256;
  // the 3D frontier's staging buffers: two per warp (dynamic shared memory)
  const size_t dyn = (MODE == 0 && JFC_RL3D_STAGE && TY * TZ <= 8)
                         ? 2 * 8 * sizeof(RlStage<TY, TZ>) + 128 : 0;
  if (dyn > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
    if (e != cudaSuccess) return e;
  }
  static int cache[64] = {0};
  int blocks = persistent_blocks_cached(cache, fn, nt, dyn);
  // (no more CTAs than find blocks: the barrier's cost grows with them)
  if constexpr (MODE == 1) blocks = std::max(1, std::min(blocks, (ts.ntiles + 63) / 64));
  if constexpr (MODE != 2) {
    static int cache_bits[64] = {0};
    const int nb = persistent_blocks_cached(cache_bits, (const void*)k_bits3<TY, TZ>, 256);
    jfc_note_launch();
    k_bits3<TY, TZ><<<(unsigned)std::min<long long>(nb, ((long long)ts.ntiles + 255) / 256), 256, 0, s>>>(ts);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  if constexpr (MODE == 0) {
    jfc_note_launch();
    const long long warps = ((long long)ts.ntiles * (TY * TZ) + 31) / 32;
    k_relabel_first<TY, TZ><<<(unsigned)((warps + 7) / 8), 256, 0, s>>>(ts);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  TileSet arg = ts;
  void* params[] = {(void*)&arg, (void*)&max_passes, (void*)&seeds};   // relabel and cut take two
  jfc_note_launch();
  const cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(nt), params, dyn, s);
  if (MODE != 0 || e != cudaSuccess || ts.cyc_mode == 0) return e;
  jfc_note_launch();
  k_end_cycle<<<1, 32, 0, s>>>(ts);
  return cudaGetLastError();
}

template <int TY, int TZ>
cudaError_t sums_t(const TileSet& ts, cudaStream_t s) {
  static int cache[64] = {0};
  const int blocks = persistent_blocks_cached(cache, (const void*)k_grid_sums<TY, TZ>, 256);
  jfc_note_launch();
  k_grid_sums<TY, TZ><<<blocks, 256, 0, s>>>(ts.d_desc, ts.d_info, ts.ntiles, ts.d_grid_sum);
  return cudaGetLastError();
}

// ---------------------------------------------------------- layout helpers
// Zero arcs that leave the grid and flag inputs the int32 solver cannot hold
// (negative capacities).
__global__ void k_fix_boundary(GridDev g, int conn, int* bad) {
  const long long total = g.plane;
  for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < total;
       n += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(n % g.pitch);
    const long long yz = n / g.pitch;
    const int y = (int)(yz % g.Hp), z = (int)(yz / g.Hp);
    const bool real = x < g.W && y < g.H && z < g.D;
    if (!real) {
      g.e[n] = 0;
      for (int k = 0; k < conn; ++k) g.r[k][n] = 0;
      g.label[n] = 0;
      continue;
    }
    bool ok[6];
    if (g.dims == 2) {
      ok[0] = x + 1 < g.W; ok[1] = y + 1 < g.H; ok[2] = y > 0; ok[3] = x > 0;
    } else {
      ok[0] = x + 1 < g.W; ok[1] = y + 1 < g.H; ok[2] = z + 1 < g.D;
      ok[3] = z > 0; ok[4] = y > 0; ok[5] = x > 0;
    }
    for (int k = 0; k < conn; ++k) {
      const int v = g.r[k][n];
      if (!ok[k]) g.r[k][n] = 0;
      else if (v < 0) *bad = 1;
    }
    g.label[n] = 0;
  }
}

__global__ void k_pack_u8(GridDev g, const uint8_t* __restrict__ src, uint8_t* __restrict__ dst) {
  const long long n = (long long)g.W * g.H * g.D;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % g.W);
    const long long yz = i / g.W;
    const int y = (int)(yz % g.H), z = (int)(yz / g.H);
    dst[i] = src[(long long)x + (long long)g.pitch * (y + (long long)g.Hp * z)];
  }
}

__global__ void k_pack_i32(GridDev g, const int* __restrict__ src, int* __restrict__ dst) {
  const long long n = (long long)g.W * g.H * g.D;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % g.W);
    const long long yz = i / g.W;
    const int y = (int)(yz % g.H), z = (int)(yz / g.H);
    dst[i] = src[(long long)x + (long long)g.pitch * (y + (long long)g.Hp * z)];
  }
}

__global__ void k_edit_tlinks(GridDev g, const uint32_t* __restrict__ idx, const int32_t* __restrict__ dcs,
                              const int32_t* __restrict__ dct, long long n, long long* dsink) {
  long long acc = 0;
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n;
       j += (long long)gridDim.x * blockDim.x) {
    const long long i = idx[j];
    const int x = (int)(i % g.W);
    const long long yz = i / g.W;
    const int y = (int)(yz % g.H), z = (int)(yz / g.H);
    const long long p = (long long)x + (long long)g.pitch * (y + (long long)g.Hp * z);
    atomicAdd(g.e + p, dcs[j] - dct[j]);
    acc += dct[j];
  }
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
  if ((threadIdx.x & 31) == 0 && acc) atomicAdd((unsigned long long*)dsink, (unsigned long long)acc);
}

}  // namespace

int persistent_blocks(const void* kernel, int threads, size_t smem) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem);
  if (per < 1) per = 1;
  return sms * per;
}

int persistent_blocks_cached(int* cache, const void* kernel, int threads, size_t smem) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return persistent_blocks(kernel, threads, smem);
  // two threads filling one entry at once compute the same value; the
  // atomic store keeps the write whole
  int v = __atomic_load_n(cache + dev, __ATOMIC_RELAXED);
  if (!v) {
    v = persistent_blocks(kernel, threads, smem);
    __atomic_store_n(cache + dev, v, __ATOMIC_RELAXED);
  }
  return v;
}

static cudaError_t bfs_dispatch(const TileSet& ts, int mode, int max_passes, const uint8_t* seeds, cudaStream_t s) {
#define JFC_BFS3(Y, Z)                                                         \
  (mode == 0 ? bfs_t<3, Y, Z, 0>(ts, max_passes, seeds, s)                     \
             : mode == 1 ? bfs_t<3, Y, Z, 1>(ts, max_passes, seeds, s) : bfs_t<3, Y, Z, 2>(ts, max_passes, seeds, s))
  if (ts.dims == 2) {
    if (mode == 0) return launch_wave_relabel(ts, s);
    if (mode == 1) return launch_wave_cut(ts, max_passes, s);
    if (ts.TR == 8) return bfs_t<2, 8, 1, 2>(ts, max_passes, seeds, s);
    if (ts.TR == 16) return bfs_t<2, 16, 1, 2>(ts, max_passes, seeds, s);
    return cudaErrorInvalidValue;
  }
  if (ts.TY == 4 && ts.TZ == 4) return JFC_BFS3(4, 4);
  if (ts.TY == 4 && ts.TZ == 2) return JFC_BFS3(4, 2);
  if (ts.TY == 16 && ts.TZ == 1) return JFC_BFS3(16, 1);
  if (ts.TY == 8 && ts.TZ == 2) return JFC_BFS3(8, 2);
  if (ts.TY == 8 && ts.TZ == 1) return JFC_BFS3(8, 1);
#undef JFC_BFS3
  return cudaErrorInvalidValue;
}

cudaError_t launch_bfs(const TileSet& ts, bool cut, int max_passes, cudaStream_t s) {
  return bfs_dispatch(ts, cut ? 1 : 0, max_passes, nullptr, s);
}

cudaError_t launch_tag(const TileSet& ts, const uint8_t* d_seeds, int max_passes, cudaStream_t s) {
  return bfs_dispatch(ts, 2, max_passes, d_seeds, s);
}

cudaError_t launch_grid_sums(const TileSet& ts, cudaStream_t s) {
  cudaError_t err = cudaMemsetAsync(ts.d_grid_sum, 0, sizeof(long long) * 2 * ts.ngrids, s);
  if (err != cudaSuccess) return err;
  if (ts.dims == 2) {
    if (ts.TR == 8) return sums_t<8, 1>(ts, s);
    if (ts.TR == 16) return sums_t<16, 1>(ts, s);
    return cudaErrorInvalidValue;
  }
  if (ts.TY == 4 && ts.TZ == 4) return sums_t<4, 4>(ts, s);
  if (ts.TY == 4 && ts.TZ == 2) return sums_t<4, 2>(ts, s);
  if (ts.TY == 16 && ts.TZ == 1) return sums_t<16, 1>(ts, s);
  if (ts.TY == 8 && ts.TZ == 2) return sums_t<8, 2>(ts, s);
  if (ts.TY == 8 && ts.TZ == 1) return sums_t<8, 1>(ts, s);
  return cudaErrorInvalidValue;
}

cudaError_t launch_mark_dirty(const TileSet& ts, cudaStream_t s) {
  // (a 3D relabel finds its frontier flags clear, unless the one before failed)
  for (int k = 0; k < 2 && ts.dims == 3; ++k) {
    const cudaError_t e = cudaMemsetAsync(ts.d_flag_bfs[k], 0, sizeof(int) * (size_t)ts.ntiles, s);
    if (e != cudaSuccess) return e;
  }
  // (no region of an earlier, failed run takes part in a cut on its own)
  for (int k = 0; k < 2 && ts.nreg > 0; ++k) {
    const cudaError_t e = cudaMemsetAsync(ts.d_rflag[k], 0, (size_t)ts.nreg, s);
    if (e != cudaSuccess) return e;
  }
  return cudaMemsetAsync(ts.d_dirty, 1, (size_t)ts.ntiles, s);
}

cudaError_t launch_clear_counters(const TileSet& ts, cudaStream_t s) {
  const cudaError_t e = cudaMemsetAsync(ts.d_ctr, 0, sizeof(DevCounters), s);
  return e == cudaSuccess ? launch_mark_dirty(ts, s) : e;
}

namespace {
__global__ void k_set_limits(DevCounters* ctr, unsigned long long polls, int h_cap) {
  ctr->spin_limit = polls;
  ctr->cyc.h_cap = h_cap;
}
}  // namespace

cudaError_t launch_set_limits(const TileSet& ts, unsigned long long polls, int h_cap, cudaStream_t s) {
  jfc_note_launch();
  k_set_limits<<<1, 1, 0, s>>>(ts.d_ctr, polls, h_cap);
  return cudaGetLastError();
}

static int grid_blocks(long long n) {
  long long b = (n + 255) / 256;
  if (b > 148 * 16) b = 148 * 16;
  if (b < 1) b = 1;
  return (int)b;
}

cudaError_t launch_fix_boundary(const GridDev& g, int conn, int* d_bad, cudaStream_t s) {
  jfc_note_launch();
  k_fix_boundary<<<grid_blocks(g.plane), 256, 0, s>>>(g, conn, d_bad);
  return cudaGetLastError();
}

cudaError_t launch_pack_labels(const GridDev& g, uint8_t* d_dense, cudaStream_t s) {
  jfc_note_launch();
  k_pack_u8<<<grid_blocks((long long)g.W * g.H * g.D), 256, 0, s>>>(g, g.label, d_dense);
  return cudaGetLastError();
}

cudaError_t launch_pack_plane(const GridDev& g, const int* d_plane, int* d_dense, cudaStream_t s) {
  jfc_note_launch();
  k_pack_i32<<<grid_blocks((long long)g.W * g.H * g.D), 256, 0, s>>>(g, d_plane, d_dense);
  return cudaGetLastError();
}

cudaError_t launch_edit_tlinks(const GridDev& g, const uint32_t* d_idx, const int32_t* d_dcs,
                               const int32_t* d_dct, size_t n, long long* d_dsink, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  jfc_note_launch();
  k_edit_tlinks<<<grid_blocks((long long)n), 256, 0, s>>>(g, d_idx, d_dcs, d_dct, (long long)n, d_dsink);
  return cudaGetLastError();
}
