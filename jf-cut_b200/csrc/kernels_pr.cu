// kernels_pr.cu — block-wise push-relabel (the JF-Cut core).
//
// Reference: graphcut_relabel_push (src/QVisualizer/cl/GraphCut/graphcut_push_relabel.cl:25-203
// for 2D, :215-439 for 3D) driven by QGCWidget::relabelPush (QGCWidget.cpp:2136-2154):
// one work-group per 16x16 / 8x8x4 tile with the tile + a one-cell halo in
// __local memory, {relabel even, relabel odd, push even, push odd} to a local
// fixpoint, boundary flow sent out with global atomics, even and odd tiles of
// the checkerboard in separate launches so adjacent tiles never run at once.
//
// B200 design:
//  * one CTA per tile of 32 x TY (x TZ) nodes, one thread per node, one warp per
//    tile row (128-byte coalesced row loads / stores); a node's excess, height
//    and residual arcs live in its thread's registers for the visit, heights
//    (with the halo) in shared memory too.  With 2D 32 x 16 relabel tiles the
//    visits work on their 32 x 8 halves (SPLIT), which keep a checkerboard
//    parity of their own;
//  * a round = one relabel step and one push step for all nodes at once
//    (two block barriers per round): each node computes its pushes and
//    gathers its neighbours';
//  * rounds repeat until a round moves nothing (__syncthreads_or) or
//    `local_iters` rounds ran; the visit then writes back only the sectors that
//    changed and sends the flow pushed across the border with global atomics;
//  * persistent cooperative launch: `sweeps` x (even tiles, odd tiles) with a
//    grid barrier between parities; each parity drains a compact device queue
//    of active tiles (one tile per CTA ticket), tiles still active re-queue
//    themselves, neighbours that received flow are queued for the other
//    parity (deduplicated).  The phase stops early when both queues are empty.
// Heights only grow between global relabels (relabel = 1 + min over residual
// arcs, applied to active nodes without an admissible arc).
#include "jfc_relax.cuh"
#include "jfc_tma.cuh"


// Iteration cap of the exact local relabel at the start of a visit (0: none).
#ifndef JFC_LOCAL_RELABEL_ITERS
#define JFC_LOCAL_RELABEL_ITERS 12
#endif

namespace {

using jfc::FULL;

template <int DIMS, int TY, int TZ>
using Tile = jfc::CtaTile<DIMS, TY, TZ>;

// Geometry of a visit's height box: 40 columns, node x at column x + 4 (the
// box the tensor copy of the halo lands in: x0 - 4 .. x0 + 35 keeps its
// first column on a 16-byte boundary).
template <int DIMS, int TY, int TZ>
using PrTile = jfc::CtaTile<DIMS, TY, TZ, 40, 4>;

// Staging buffer of one visit:
// the tile's planes {e, h, r[0..K-1]} (plane-major, thread order), as they were
// when the visit began, and the h plane over the tile plus its one-cell halo.
template <int DIMS, int TY, int TZ>
struct alignas(128) PrStage {
  using T = PrTile<DIMS, TY, TZ>;
  static constexpr int P = 2 + T::K;
  static constexpr unsigned kBytes = (unsigned)(sizeof(int) * (P * T::NT + T::HN));   // bytes one fill copies
  int pl[P][T::NT];
  int hb[T::HN];
};

template <int DIMS, int TY, int TZ>
struct PrSmem {
  using T = PrTile<DIMS, TY, TZ>;
  int d[2 * (T::D - 1)][T::NT];   // a round's pushes along +y, -y (, +z, -z)
  unsigned run[2 * (T::D - 1)][T::R];   // (local relabel) per tile row: nodes with a residual arc +y, -y (, +z, -z)
  int tile;
  int4 ti;                // its tile: {grid, x, y, z}
  int buf;                // staging buffer of the item being visited
  int gen;                // worklist: generation of the item being visited
  int face[6];            // any flow left through face: x-, x+, y-, y+, z-, z+
  int q_nb[6];            // after a visit: the work item behind each face that received flow, or -1
  int active;             // after a visit: the item still holds an active node
  int local_iters;        // rounds of a visit, at most
};

template <int DIMS, int TY, int TZ>
__device__ __forceinline__ void halo_cell(int c, int& x, int& y, int& z, int& face) {
  Tile<DIMS, TY, TZ>::halo_cell(c, x, y, z, face);
}

// SPLIT: the work item `tid` is half `tid & 1` (rows 0-7 / 8-15) of the 2D
// 32x16 tile `tid >> 1`, visited as a 32x8 tile; the halves keep their own
// checkerboard parity, so the two halves of a tile never run at once.
// Coordinates of work item `tid`: {grid, tile x, y, z} of its tile.  A set of
// one grid computes them (a table look-up is a round trip to L2 in front of
// the copies of the tile).
template <bool SPLIT>
__device__ __forceinline__ int4 item_tile(const TileSet& ts, int tid) {
  const int tile = SPLIT ? tid >> 1 : tid;
  if (ts.ngrids != 1) return ts.d_info[tile];
  const GridDev& g = ts.d_desc[0];
  const unsigned row = (unsigned)tile / (unsigned)g.tiles_x;
  return make_int4(0, tile - (int)row * g.tiles_x, (int)(row % (unsigned)g.tiles_y), (int)(row / (unsigned)g.tiles_y));
}

// The work item behind face f of item `tid` (x-, x+, y-, y+, z-, z+; ti: its
// tile), -1 where the face is the grid's border.
template <int DIMS, int TY, int TZ, bool SPLIT>
__device__ __forceinline__ int face_item(const TileSet& ts, int tid, const int4& ti, int f) {
  const int tile = SPLIT ? tid >> 1 : tid, half = SPLIT ? tid & 1 : 0;
  const GridDev& g = ts.d_desc[ti.x];
  const int txs = g.tiles_x, tys = g.tiles_y, tzs = g.tiles_z;
  switch (f) {
    case 0: return ti.y > 0 ? (SPLIT ? tid - 2 : tid - 1) : -1;
    case 1: return ti.y < txs - 1 ? (SPLIT ? tid + 2 : tid + 1) : -1;
    case 2: return SPLIT ? (half ? tid - 1 : (ti.z > 0 ? 2 * (tile - txs) + 1 : -1)) : (ti.z > 0 ? tid - txs : -1);
    case 3: return SPLIT ? (half ? (ti.z < tys - 1 ? 2 * (tile + txs) : -1) : tid + 1)
                         : (ti.z < tys - 1 ? tid + txs : -1);
    case 4: return DIMS == 3 && ti.w > 0 ? tid - txs * tys : -1;
    case 5: return DIMS == 3 && ti.w < tzs - 1 ? tid + txs * tys : -1;
    default: return -1;
  }
}

// Grid and origin (elements) of work item `tid` in tile ti.
template <int DIMS, int TY, int TZ, bool SPLIT>
__device__ __forceinline__ int4 item_origin(int tid, const int4& ti) {
  const int half = SPLIT ? tid & 1 : 0;
  return make_int4(ti.x, ti.y * 32, SPLIT ? (2 * ti.z + half) * TY : ti.z * TY, ti.w * TZ);
}

// Fill staging buffer `st` with work item `tid` by two tensor copies (the
// tile's planes, and the h plane over the tile and its halo), completed on
// `bar`.  Issued by one thread.  Box cells outside the grid arrive as zeros;
// the visit sets the halo ones to INF.
template <int DIMS, int TY, int TZ, bool SPLIT>
__device__ __forceinline__ void pr_stage_issue(const TileSet& ts, int tid, const int4& ti, PrStage<DIMS, TY, TZ>& st,
                                               uint64_t* bar, int& acquired_grid) {
  const int4 o = item_origin<DIMS, TY, TZ, SPLIT>(tid, ti);
  const char* maps = (const char*)ts.d_tmap + (size_t)o.x * 384;   // three maps per grid
  if (o.x != acquired_grid) {
    jfc::fence_tmap_acquire(maps);
    jfc::fence_tmap_acquire(maps + 128);
    acquired_grid = o.x;
  }
  jfc::fence_async_shared();   // the buffer's previous visit wrote it through the generic proxy
  jfc::mbar_arrive_tx(bar, PrStage<DIMS, TY, TZ>::kBytes);
  jfc::tma_load_4d(&st.pl[0][0], maps, o.y, o.z, o.w, 0, bar);
  jfc::tma_load_3d(&st.hb[0], maps + 128, o.y - 4, o.z - 1, DIMS == 3 ? o.w - 1 : 0, bar);
}

// In-tile distances d(u) = min(d(v) + 1) over residual arcs u -> v, 0 at
// deficits, the halo's heights fixed, to the fixpoint (false when it takes
// more than JFC_LOCAL_RELABEL_ITERS iterations).  An iteration closes the rows
// along runs of residual arcs (both directions at once, by doubling shuffles:
// a path that turns back inside a row is never shorter), publishes the values
// and closes columns (and z lines) from what the other rows published, as far
// as this node's runs of residual arcs go.  One barrier per iteration, which
// also tells whether the rows changed anything since the last publication; if
// not, nothing can.  4 iterations on average.  Closing lines through shared
// memory, the two directions one after the other, with two barriers an
// iteration, took 4,900-5,500 cycles per visit, this 3,400 (3D) to 4,800
// (push-relabel of a 2560 x 1440 x 50 video 54.4 -> 51.0 ms).
template <class T, class Smem>
__device__ __forceinline__ bool local_distance(Smem& s, const int* sh, int hi, const int (&r)[T::K], int e, int x, int y,
                                               int z, int row, int& dist) {
  constexpr int TY = T::TY, TZ = T::TZ;
  const int t = threadIdx.x;
  const unsigned xp = __ballot_sync(FULL, r[T::XP] > 0) & 0x7fffffffu, xm = __ballot_sync(FULL, r[T::XM] > 0) & ~1u;
  const unsigned yp = __ballot_sync(FULL, r[T::YP] > 0), ym = __ballot_sync(FULL, r[T::YM] > 0);
  unsigned zp = 0, zm = 0;
  if constexpr (T::D == 3) {
    zp = __ballot_sync(FULL, r[T::ZP] > 0);
    zm = __ballot_sync(FULL, r[T::ZM] > 0);
  }
  if (x == 0) {
    s.run[0][row] = yp;
    s.run[1][row] = ym;
    if constexpr (T::D == 3) {
      s.run[2][row] = zp;
      s.run[3][row] = zm;
    }
  }
  // the halo is folded in once
  int v = e < 0 ? 0 : JFC_INF;
  if (r[T::XP] > 0 && x == 31) v = min(v, sh[hi + 1] + 1);
  if (r[T::XM] > 0 && x == 0) v = min(v, sh[hi - 1] + 1);
  if (r[T::YP] > 0 && y == TY - 1) v = min(v, sh[hi + T::SY] + 1);
  if (r[T::YM] > 0 && y == 0) v = min(v, sh[hi - T::SY] + 1);
  if constexpr (T::D == 3) {
    if (r[T::ZP] > 0 && z == TZ - 1) v = min(v, sh[hi + T::SZ] + 1);
    if (r[T::ZM] > 0 && z == 0) v = min(v, sh[hi - T::SZ] + 1);
  }
  // run lengths of residual arcs from this node, inside the tile
  const int right = __ffs(~(xp >> x)) - 1;                     // (bit 31 of xp is 0)
  const int left = __clz(~(xm << (31 - x)));                   // (bit 0 of xm is 0)
  int up = 0, down = 0, back = 0, front = 0;                   // -y, +y, -z, +z
  int old = JFC_INF + 1;                                       // (no value: the first publication counts as a change)
  for (int it = 0; it < JFC_LOCAL_RELABEL_ITERS; ++it) {
    int a = v, b = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int na = __shfl_down_sync(FULL, a, off), nb = __shfl_up_sync(FULL, b, off);
      if (right >= off) a = min(a, na + off);
      if (left >= off) b = min(b, nb + off);
    }
    v = min(a, b);
    int* pub = s.d[it & 1];
    pub[t] = v;
    if (!__syncthreads_or(v != old)) {
      dist = v;
      return true;
    }
    if (it == 0) {
      bool u = true, d = true;
#pragma unroll
      for (int k = 0; k < TY - 1; ++k) {
        d = d && y + k < TY - 1 && (s.run[0][row + k < T::R ? row + k : row] >> x & 1u);
        u = u && y - k > 0 && (s.run[1][row >= k ? row - k : row] >> x & 1u);
        down += d;
        up += u;
      }
      if constexpr (T::D == 3) {
        bool f = true, c = true;
#pragma unroll
        for (int k = 0; k < TZ - 1; ++k) {
          f = f && z + k < TZ - 1 && (s.run[2][row + k * TY < T::R ? row + k * TY : row] >> x & 1u);
          c = c && z - k > 0 && (s.run[3][row >= k * TY ? row - k * TY : row] >> x & 1u);
          front += f;
          back += c;
        }
      }
    }
    old = v;
#pragma unroll
    for (int k = 1; k < TY; ++k) {
      if (k <= down) v = min(v, pub[t + 32 * k] + k);
      if (k <= up) v = min(v, pub[t - 32 * k] + k);
    }
    if constexpr (T::D == 3) {
#pragma unroll
      for (int k = 1; k < TZ; ++k) {
        if (k <= front) v = min(v, pub[t + 32 * TY * k] + k);
        if (k <= back) v = min(v, pub[t - 32 * TY * k] + k);
      }
    }
  }
  return false;
}

// One visit of work item `tid` (in tile ti) on staging buffer `st`; staged: the
// tensor copies already filled it, otherwise the visit loads the tile itself.
// failed: a staging copy never completed for this thread; the visit then
// returns -1 to every thread of the CTA and changes nothing.  On
// return s.active tells whether the item still holds an active node and
// s.q_nb[f] the item behind each face f that received flow (-1: none).  The
// caller queues them.
template <int DIMS, int TY, int TZ, bool SPLIT>
__device__ __forceinline__ int pr_visit(const TileSet& ts, int tid, const int4& ti, bool local_relabel,
                                        PrSmem<DIMS, TY, TZ>& s, PrStage<DIMS, TY, TZ>& st, bool staged, bool failed) {
  using T = PrTile<DIMS, TY, TZ>;
  const int t = threadIdx.x;
  const int x = t & 31, row = t >> 5, y = row % TY, z = row / TY;
  const int4 o = item_origin<DIMS, TY, TZ, SPLIT>(tid, ti);
  const GridDev& g = ts.d_desc[o.x];
  const int pitch = g.pitch;
  const long long slab = (long long)g.pitch * g.Hp;
  const int x0 = o.y, y0 = o.z, z0 = o.w;
  const long long tbase = (long long)x0 + (long long)y0 * pitch + (long long)z0 * slab;
  const long long n = tbase + x + (long long)y * pitch + (long long)z * slab;
  const int hi = T::hidx(x, y, z);
  int* const sh = st.hb;
  JFC_PCLK_DECL

  // ---- the tile and its halo heights
  if (!staged) {
    st.pl[0][t] = g.e[n];
    st.pl[1][t] = g.h[n];
#pragma unroll
    for (int k = 0; k < T::K; ++k) st.pl[2 + k][t] = g.r[k][n];
  }
  const int e0 = st.pl[0][t], h0 = st.pl[1][t];
  int r0[T::K];
#pragma unroll
  for (int k = 0; k < T::K; ++k) r0[k] = st.pl[2 + k][t];
  for (int c = t; c < T::NHALO; c += T::NT) {
    int hx, hy, hz, f;
    halo_cell<DIMS, TY, TZ>(c, hx, hy, hz, f);
    const int gx = x0 + hx, gy = y0 + hy, gz = z0 + hz;
    const bool in = gx >= 0 && gx < pitch && gy >= 0 && gy < g.Hp && gz >= 0 && gz < g.Dp;
    if (!staged || !in)
      sh[T::hidx(hx, hy, hz)] = in ? g.h[(long long)gx + (long long)gy * pitch + (long long)gz * slab] : JFC_INF;
  }
  if (t < 6) s.face[t] = 0;
  if (__syncthreads_or(failed)) return -1;
  JFC_PCLK(ts.d_ctr, 0);
  // the node's own height lives in a register (only its owner writes it); the
  // shared copy is what the neighbours read
  int hown = h0;
  if (JFC_LOCAL_RELABEL_ITERS > 0 && local_relabel) {
    // local relabel: distance to the nearest in-tile deficit or halo node
    // over residual arcs (halo heights fixed), then h = max(h, distance).
    // The pointwise max of two valid labellings is valid, so heights stay
    // monotone (push-relabel termination holds) while excess trapped in the
    // tile jumps straight to INF instead of climbing one level per round.
    // A partial relaxation overestimates distances, so the labelling is only
    // applied when the in-tile fixpoint was reached.
    int dist = 0;
    if (local_distance<T>(s, sh, hi, r0, e0, x, y, z, row, dist)) hown = max(dist, h0);
#ifdef JFC_PHASE_CLOCK
    if (threadIdx.x == 0 && hown != h0) atomicAdd(&ts.d_ctr->prof[5], 1ull);
#endif
  }
  sh[hi] = hown;
  __syncthreads();
  JFC_PCLK(ts.d_ctr, 1);

  // Rounds, the node's excess, height and arcs in registers.  A push u -> v is
  // computed by u and gathered by v: along x by shuffles (a warp holds a tile
  // row), along y and z through s.d.  Under one height vector two neighbours
  // never push to each other, so a node's arc changes by its own push or by
  // its neighbour's.  Nothing diverges and nothing is atomic; a round is a
  // chain of two block barriers and about 60 instructions per thread, 610-740
  // cycles.  With the state in shared memory and the pushes as divergent
  // shared-memory reductions a round took 1,000-1,230 cycles (push-relabel of
  // a 15000 x 10000 solve 38.5 -> 33.4 ms, of a 2560 x 1440 x 50 video 60.9 ->
  // 54.4 ms).
  int e = e0, r[T::K], hn[T::K];
#pragma unroll
  for (int k = 0; k < T::K; ++k) r[k] = r0[k];
  const int h_left = sh[hi - 1], h_right = sh[hi + 1];   // (halo cells for lanes 0 and 31)
  auto heights = [&]() {
    const int hr = __shfl_down_sync(FULL, hown, 1), hl = __shfl_up_sync(FULL, hown, 1);
    hn[T::XP] = x == 31 ? h_right : hr;
    hn[T::XM] = x == 0 ? h_left : hl;
    hn[T::YP] = sh[hi + T::SY];
    hn[T::YM] = sh[hi - T::SY];
    if constexpr (DIMS == 3) {
      hn[T::ZP] = sh[hi + T::SZ];
      hn[T::ZM] = sh[hi - T::SZ];
    }
  };
  heights();
  __syncthreads();   // (the first round's relabels write what the other warps read here)
  // push order: +x, +y, -y, (+z, -z,) -x
  constexpr int kOrder[6] = {T::XP, T::YP, T::YM, DIMS == 3 ? T::ZP : T::XM, T::ZM, T::XM};
  constexpr int NP = T::K;
  int it = 0;
  for (; it < s.local_iters; ++it) {
    // relabel every active node without an admissible arc
    // (graphcut_push_relabel.cl:80-99 relabels two colours in turn): 1 + the
    // lowest residual neighbour; heights only grow, so the labelling stays
    // valid when neighbours do so at once
    const bool act = e > 0 && hown < JFC_INF;
    bool adm = false;
    int m = JFC_INF;
#pragma unroll
    for (int k = 0; k < T::K; ++k) {
      adm |= r[k] > 0 && hn[k] == hown - 1;
      m = min(m, r[k] > 0 ? hn[k] : JFC_INF);
    }
    bool did = act && !adm;
    if (did) {
      hown = max(hown, min(m + 1, JFC_INF));
      sh[hi] = hown;
    }
    __syncthreads();
    heights();
    // push along admissible arcs in the reference's order
    int left = act && hown < JFC_INF ? e : 0, d[T::K];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      const int k = kOrder[q == NP - 1 ? 5 : q];
      d[k] = hn[k] == hown - 1 ? min(left, r[k]) : 0;
      left -= d[k];
    }
    s.d[0][t] = d[T::YP];
    s.d[1][t] = d[T::YM];
    if constexpr (DIMS == 3) {
      s.d[2][t] = d[T::ZP];
      s.d[3][t] = d[T::ZM];
    }
    int in[T::K], out = 0;   // in[k]: pushed to this node by its neighbour in direction k
    in[T::XP] = __shfl_down_sync(FULL, d[T::XM], 1);
    in[T::XM] = __shfl_up_sync(FULL, d[T::XP], 1);
    if (x == 31) in[T::XP] = 0;
    if (x == 0) in[T::XM] = 0;
#pragma unroll
    for (int k = 0; k < T::K; ++k) out += d[k];
    did |= out != 0;
    if (!__syncthreads_or(did)) break;
    in[T::YP] = y < TY - 1 ? s.d[1][t + 32] : 0;
    in[T::YM] = y > 0 ? s.d[0][t - 32] : 0;
    if constexpr (DIMS == 3) {
      in[T::ZP] = z < TZ - 1 ? s.d[3][t + 32 * TY] : 0;
      in[T::ZM] = z > 0 ? s.d[2][t - 32 * TY] : 0;
    }
    e -= out;
#pragma unroll
    for (int k = 0; k < T::K; ++k) {
      e += in[k];
      r[k] += in[k] - d[k];
    }
  }
  const int rounds = it < s.local_iters ? it + 1 : s.local_iters;
  JFC_PCLK(ts.d_ctr, 2);

  // ---- write back the 32-byte sectors of each row that hold a changed word
  //      (nothing else writes the tile while it is visited, so the unchanged
  //      words of a sector are rewritten with their own values)
  const int e1 = e, h1 = hown;
  {
    const int grp = x & ~7;
    auto put = [&](int* gplane, int v, bool changed) {
      if ((__ballot_sync(FULL, changed) >> grp) & 0xFFu) gplane[n] = v;
    };
    put(g.e, e1, e1 != st.pl[0][t]);
    put(g.h, h1, h1 != st.pl[1][t]);
#pragma unroll
    for (int k = 0; k < T::K; ++k) put(g.r[k], r[k], r[k] != st.pl[2 + k][t]);
  }
  // ---- send the flow pushed across the border into the neighbours' excess
  //      and reverse arcs: what a border arc lost (arcs leaving the grid are
  //      zero, so only neighbours inside it can receive flow)
  auto send = [&](bool border, int k, int face, long long off) {
    const int v = border ? st.pl[2 + k][t] - r[k] : 0;
    if (v) {
      atomicAdd(g.e + n + off, v);
      atomicAdd(g.r[T::K - 1 - k] + n + off, v);
      s.face[face] = 1;
    }
  };
  send(x == 0, T::XM, 0, -1);
  send(x == 31, T::XP, 1, 1);
  send(y == 0, T::YM, 2, -(long long)pitch);
  send(y == TY - 1, T::YP, 3, pitch);
  if constexpr (DIMS == 3) {
    send(z == 0, T::ZM, 4, -slab);
    send(z == TZ - 1, T::ZP, 5, slab);
  }
  const bool active = __syncthreads_or((e1 > 0) & (h1 < JFC_INF));
  // flow crossed face f only toward an item inside the grid (arcs leaving
  // the grid are zero)
  if (t < 6) {
    const int nb = s.face[t] ? face_item<DIMS, TY, TZ, SPLIT>(ts, tid, ti, t) : -1;
    s.q_nb[t] = nb;
    // the global relabel reads the arcs and signs of these tiles again
    if (nb >= 0) ts.d_dirty[SPLIT ? nb >> 1 : nb] = 1;
  }
  if (t == 0) {
    s.active = active ? 1 : 0;
    ts.d_dirty[SPLIT ? tid >> 1 : tid] = 1;
  }
  __syncthreads();
  JFC_PCLK(ts.d_ctr, 3);
  return rounds;
}

// Persistent push-relabel phase: 2*sweeps alternating parity sweeps separated
// by grid barriers.  Sweep s of parity p drains queue q_pr[p][cur[p]], a CTA's
// first item at its block index, the others by ticket; tiles still active go
// to q_pr[p][1-cur], neighbours that received flow to the other parity's
// pending buffer.
//
// In the tail of a solve a sweep holds a few items and its time is a chain of
// latencies, so the chain is kept short: which buffer a parity is on follows
// from the sweep index; the queue's length and the CTA's own entry are one
// round trip to L2; the barrier is one growing counter (pr_bar, zeroed with
// the tickets by the relabel before) whose arrivals are also its release; the
// counters that a sweep leaves are reset by block 0 during the next one.
// 26 us a sweep before, 19.5 now (4096 x 3072, 200-1,000 active tiles).
//
// Staging (ts.d_tmap set): tensor copies fill one of two staging buffers in
// dynamic shared memory.  While a visit runs, the CTA's next ticket is
// already being copied into the other buffer, as long as the sweep holds at
// least a grid's worth of tickets beyond the current one (in a short sweep
// a second ticket would only keep another CTA idle).  A prefetched item is
// safe to read early: items of one sweep are never adjacent, so nothing
// writes its tile or its halo heights until the sweep ends.
// CTAs per SM the phase is compiled for (its registers): the 2D 32 x 8 form
// JFC_PR2D_MINB, other 256-node tiles 3, 512-node tiles 2
#ifndef JFC_PR2D_MINB
#define JFC_PR2D_MINB 4
#endif
template <int DIMS, int TY, int TZ, bool SPLIT>
__global__ void __launch_bounds__(Tile<DIMS, TY, TZ>::NT,
                                  (DIMS == 2 && TY == 8) ? JFC_PR2D_MINB : Tile<DIMS, TY, TZ>::NT > 256 ? 2 : 3)
    k_pr_phase(TileSet ts, int sweeps, int local_iters) {
  using Stage = PrStage<DIMS, TY, TZ>;
  __shared__ PrSmem<DIMS, TY, TZ> sm;
  __shared__ uint64_t s_bar[2];
  extern __shared__ __align__(128) unsigned char s_dyn[];
  Stage* stage = reinterpret_cast<Stage*>(s_dyn + ((128u - (jfc::smem_addr(s_dyn) & 127u)) & 127u));
  DevCounters* ctr = ts.d_ctr;
  const bool tma = ts.d_tmap != nullptr;
  unsigned long long visits = 0, rounds = 0;
  const unsigned long long t0 = jfc::global_ns();
  const unsigned long long cap = jfc::spin_cap(ctr);
  if (tma && threadIdx.x == 0) {
    jfc::mbar_init(&s_bar[0], 1);
    jfc::mbar_init(&s_bar[1], 1);
    jfc::fence_mbar_init();
  }
  __syncthreads();
  unsigned parity = 0;      // bit b: phase parity of buffer b's next fill
  int acquired_grid = -1;   // thread 0: grid whose tensor maps it acquired
  int next_buf = 0;         // thread 0: buffer of the next fill
  int s = 0;
  const int npairs = sweeps > 0 ? sweeps : jfc::vload(&ctr->cyc.pr_sweeps);
  if (jfc::cycle_skips(ts)) return;
  if (threadIdx.x == 0) sm.local_iters = sweeps > 0 ? local_iters : jfc::vload(&ctr->cyc.local_iters);
  const int own = min((int)blockIdx.x, ts.ntiles - 1);   // (a parity's queue holds at most ntiles items)
  int cur[2] = {0, 0};   // pending buffer per parity (0 after a global relabel)
  bool failed = false;   // a staging copy never completed (error raised): leave
  for (; s < 2 * npairs; ++s) {
    const int p = s & 1, b = cur[p], bo = cur[p ^ 1];
    int* const queue = ts.d_q_pr[p][b];
    const int n = jfc::vload(&ctr->qn_pr[p][b]), n_other = jfc::vload(&ctr->qn_pr[p ^ 1][bo]);
    const int mine = jfc::vload(queue + own);
    if (n == 0 && n_other == 0) break;   // nothing left anywhere
    if (threadIdx.x == 0) {
      // the previous sweep's writes (seen through the grid barrier) come before
      // this sweep's tensor reads
      if (tma) jfc::fence_async_global();
      if (blockIdx.x == 0) {
        // what the previous sweep used up: next touched after this sweep's barrier
        ctr->ticket[p ^ 1] = 0;
        if (s > 0) ctr->qn_pr[p ^ 1][bo ^ 1] = 0;
      }
    }
    int pre = -1, pre_buf = 0;   // thread 0: the prefetched item, its tile and its buffer
    int4 pre_ti = make_int4(0, 0, 0, 0);
    long long k = blockIdx.x;    // thread 0: ticket of the current item
    bool more = (long long)blockIdx.x < n;
    for (bool first = true; more; first = false) {
      if (threadIdx.x == 0) {
        int item = -1, buf = 0;
        int4 ti = make_int4(0, 0, 0, 0);
        auto issue = [&](int it, const int4& t4) {
          const int bf = next_buf;
          ts.d_flag_pr[it] = 0;
          if (tma) {
            next_buf ^= 1;
            pr_stage_issue<DIMS, TY, TZ, SPLIT>(ts, it, t4, stage[bf], &s_bar[bf], acquired_grid);
            return bf;
          }
          return 0;
        };
        auto next_ticket = [&]() { return (long long)gridDim.x + atomicAdd(&ctr->ticket[p], 1u); };
        if (pre >= 0) {
          item = pre; ti = pre_ti; buf = pre_buf; pre = -1;
        } else {
          if (!first) k = next_ticket();
          if (k < n) {
            item = first ? mine : queue[k];
            ti = item_tile<SPLIT>(ts, item);
            buf = issue(item, ti);
          }
        }
        if (tma && item >= 0 && k + gridDim.x < n) {
          const long long k2 = next_ticket();
          if (k2 < n) {
            pre = queue[k2];
            pre_ti = item_tile<SPLIT>(ts, pre);
            k = k2;
            pre_buf = issue(pre, pre_ti);
          }
        }
        sm.tile = item;
        sm.ti = ti;
        sm.buf = buf;
      }
      __syncthreads();
      const int tid = sm.tile, buf = sm.buf;
      const int4 ti = sm.ti;
      if (tid < 0) break;
      bool late = false;
      if (tma) {
        late = !jfc::mbar_wait(&s_bar[buf], (parity >> buf) & 1u, cap);
        parity ^= 1u << buf;
      }
      // first sweep of a phase: nothing moved since the exact global relabel
      // (the halo tiles have the other parity), so the local relabel would
      // reproduce the heights it finds
      const int rd = pr_visit<DIMS, TY, TZ, SPLIT>(ts, tid, ti, s > 0, sm, stage[buf], tma, late);
      if (rd < 0) {
        if (threadIdx.x == 0) {
          atomicExch(&ctr->error, 1);
          // copies still in flight land before the CTA leaves its shared
          // memory: bounded by a fixed poll count of its own, not by the
          // (possibly tiny) spin limit that gave up above
          constexpr unsigned long long kDrainPolls = 1ull << 26;
          jfc::mbar_wait(&s_bar[buf], ((parity >> buf) & 1u) ^ 1u, kDrainPolls);
          if (pre >= 0) jfc::mbar_wait(&s_bar[pre_buf], (parity >> pre_buf) & 1u, kDrainPolls);
        }
        failed = true;
        break;
      }
      rounds += rd;
      ++visits;
      // queue: neighbours for the other parity (lanes 0-5), myself for my
      // parity's next sweep (lane 6), both counters at once
      if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        const int nb = lane < 6 ? sm.q_nb[lane] : -1;
        bool won = false;
        if (nb >= 0) won = atomicExch(ts.d_flag_pr + nb, 1) == 0;
        if (lane == 6 && sm.active) {
          ts.d_flag_pr[tid] = 1;
          won = true;
        }
        const unsigned m = __ballot_sync(FULL, won), mn = m & 63u;
        int at = 0;
        if (lane == 0 && mn) at = atomicAdd(&ctr->qn_pr[p ^ 1][bo], __popc(mn));
        if (lane == 6 && won) at = atomicAdd(&ctr->qn_pr[p][b ^ 1], 1);
        const int at0 = __shfl_sync(FULL, at, 0);
        if (won) {
          if (lane == 6) ts.d_q_pr[p][b ^ 1][at] = tid;
          else ts.d_q_pr[p ^ 1][bo][at0 + __popc(mn & ((1u << lane) - 1u))] = nb;
        }
      }
      more = n > (int)gridDim.x;   // otherwise every item had its CTA
      if (more) __syncthreads();
    }
    if (failed) break;
    cur[p] = b ^ 1;
    JFC_PCLK_DECL
    const bool ok = jfc::arrive_wait(ctr, &ctr->pr_bar, (unsigned long long)(s + 1) * gridDim.x);
    JFC_PCLK(ctr, 4);
    if (!ok) break;
  }
  if (threadIdx.x == 0) {
    if (visits) atomicAdd(&ctr->visits, visits);
    if (rounds) atomicAdd(&ctr->rounds, rounds);
    if (blockIdx.x == 0) {
      ctr->sweeps_done = s;
      ctr->ns_pr += jfc::global_ns() - t0;
    }
  }
}

// ---------------------------------------------------------------------------
// Asynchronous push-relabel phase: a worklist instead of parity sweeps.
//
// The sweeps keep adjacent work items apart by running one checkerboard
// colour at a time, with a grid barrier between colours; in the tail of a
// solve a sweep holds a few items and every CTA waits at the barrier for the
// slowest visit.  Here the items live in a ring (one entry per queued item:
// the queued flags dedupe), any free CTA takes the next entry, and adjacency
// is kept apart by per-item locks instead: a visit takes its item's lock,
// then (after a sequentially consistent fence) checks that no item behind
// its faces holds one; of two adjacent items that try at once at least one
// sees the other and backs off (the entry goes back to the ring).  So a visit
// sees exactly what it would see in a sweep: its item and halo untouched by
// any other visit while it runs.  An entry carries a generation that plays
// the role of the sweep index: a visit of generation k queues the items it
// fed for k + 1 (the other colour's next sweep) and itself for k + 2 (its own
// colour's next sweep), and a phase of `npairs` sweep pairs visits
// generations 0 .. 2 * npairs - 1 (the sweeps' budget); items past it stay
// active for the next global relabel.  The phase ends when
// no queued item is left (every wait is bounded, see jfc::spin_cap).
constexpr unsigned long long kRingEmpty = ~0ull;

__device__ __forceinline__ unsigned long long ring_entry(int item, int gen) {
  return ((unsigned long long)(unsigned)gen << 32) | (unsigned)item;
}

// Put one entry into the ring (a position reserved at the tail; the slot is
// free, or freed by its reader within a few polls).  Returns false after an
// error.
__device__ __forceinline__ bool pr_ring_put(unsigned long long* ring, unsigned cap, unsigned* tail, int* err,
                                            unsigned long long max_spins, unsigned long long v) {
  const unsigned pos = atomicAdd(tail, 1u);
  unsigned long long* slot = ring + pos % cap;
  unsigned long long spins = 0;
  while (atomicCAS(slot, kRingEmpty, v) != kRingEmpty) {
    if (++spins > max_spins || jfc::vload(err)) { atomicExch(err, 1); return false; }
    __nanosleep(32);
  }
  return true;
}

template <int DIMS, int TY, int TZ, bool SPLIT>
__global__ void __launch_bounds__(Tile<DIMS, TY, TZ>::NT)
    k_pr_async(TileSet ts, int sweeps, int local_iters) {
  __shared__ PrSmem<DIMS, TY, TZ> sm;
  extern __shared__ __align__(128) unsigned char s_dyn[];
  PrStage<DIMS, TY, TZ>& stage =
      *reinterpret_cast<PrStage<DIMS, TY, TZ>*>(s_dyn + ((128u - (jfc::smem_addr(s_dyn) & 127u)) & 127u));
  DevCounters* ctr = ts.d_ctr;
  const unsigned long long t0 = jfc::global_ns();
  const int npairs = sweeps > 0 ? sweeps : jfc::vload(&ctr->cyc.pr_sweeps);
  if (jfc::cycle_skips(ts)) return;
  if (threadIdx.x == 0) sm.local_iters = sweeps > 0 ? local_iters : jfc::vload(&ctr->cyc.local_iters);
  const int gens = 2 * npairs;
  const unsigned cap = (unsigned)(SPLIT ? 2 * ts.ntiles : ts.ntiles);
  unsigned long long* ring = ts.d_pr_ring;
  int* lock = ts.d_pr_lock;
  // ---- the ring starts with the items the global relabel queued (both
  //      parity queues, colour 0 first: the first wave of takers is
  //      conflict-free), generation 0; locks clear
  const int b0 = jfc::vload(&ctr->cur_pr[0]), b1 = jfc::vload(&ctr->cur_pr[1]);
  const int n0 = jfc::vload(&ctr->qn_pr[0][b0]), n1 = jfc::vload(&ctr->qn_pr[1][b1]);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < cap; i += (long long)gridDim.x * blockDim.x) {
    unsigned long long v = kRingEmpty;
    if (i < n0) v = ring_entry(ts.d_q_pr[0][b0][i], 0);
    else if (i < n0 + n1) v = ring_entry(ts.d_q_pr[1][b1][i - n0], 0);
    ring[i] = v;
    lock[i] = 0;
  }
  const bool ok = jfc::grid_sync(ctr, [&]() {
    ctr->pr_head = 0;
    ctr->pr_tail = (unsigned)(n0 + n1);
    ctr->pr_out = n0 + n1;
    ctr->sweeps_done = 0;
  });
  const unsigned long long max_spins = jfc::spin_cap(ctr);
  unsigned long long visits = 0, rounds = 0;
  int maxgen = -1;
  while (ok) {
    if (threadIdx.x == 0) {
      int item = -1, gen = 0;
      const unsigned k = atomicAdd(&ctr->pr_head, 1u);
      unsigned long long* slot = ring + k % cap;
      // bounded: the entry arrives, or no item is left, or an error; the
      // count restarts whenever the worklist moves
      unsigned long long spins = 0, v = kRingEmpty;
      unsigned seen_tail = (unsigned)jfc::vload((const int*)&ctr->pr_tail);
      int seen_out = jfc::vload(&ctr->pr_out);
      for (;;) {
        if (*(volatile unsigned long long*)slot != kRingEmpty) {
          v = atomicExch(slot, kRingEmpty);
          if (v != kRingEmpty) break;
        }
        const int out = jfc::vload(&ctr->pr_out);
        if (out == 0 || jfc::vload(&ctr->error)) break;
        const unsigned tl = (unsigned)jfc::vload((const int*)&ctr->pr_tail);
        if (out != seen_out || tl != seen_tail) {
          seen_out = out;
          seen_tail = tl;
          spins = 0;
        } else if (++spins > max_spins) {
          atomicExch(&ctr->error, 1);
          break;
        }
        __nanosleep(32);
      }
      if (v != kRingEmpty) {
        item = (int)(unsigned)(v & 0xffffffffu);
        gen = (int)(v >> 32);
        // neighbour exclusion (see above)
        const int4 ti = item_tile<SPLIT>(ts, item);
        sm.ti = ti;
        bool conflict = atomicCAS(lock + item, 0, 1) != 0;
        if (!conflict) {
          asm volatile("fence.sc.gpu;" ::: "memory");
#pragma unroll
          for (int f = 0; f < (DIMS == 3 ? 6 : 4); ++f) {
            const int nb = face_item<DIMS, TY, TZ, SPLIT>(ts, item, ti, f);
            if (nb >= 0 && jfc::vload(lock + nb) != 0) conflict = true;
          }
          if (conflict) atomicExch(lock + item, 0);
        }
        if (conflict) {
          // back to the ring, same generation, still flagged as queued (it
          // stays outstanding); -2: take the next entry
          if (!pr_ring_put(ring, cap, &ctr->pr_tail, &ctr->error, max_spins, v)) item = -1;
          else item = -2;
        } else {
          ts.d_flag_pr[item] = 0;   // dequeued: a neighbour may queue it again once we unlock
          __threadfence();
        }
      }
      sm.tile = item;
      sm.gen = gen;
    }
    __syncthreads();
    const int item = sm.tile, gen = sm.gen;
    if (item == -1) break;
    if (item == -2) {
      __syncthreads();   // sm.tile is rewritten only after every thread read it
      continue;
    }
    // generation 0: nothing around the item moved since the exact global
    // relabel unless a neighbour was visited first; the local relabel is an
    // improvement only, so skipping it is safe either way
    rounds += pr_visit<DIMS, TY, TZ, SPLIT>(ts, item, sm.ti, gen > 0, sm, stage, false, false);
    ++visits;
    maxgen = max(maxgen, gen);
    // release the item (its writes visible first), then queue what it fed
    // and itself for generation gen + 1, then count it done
    if (threadIdx.x == 0) {
      __threadfence();
      atomicExch(lock + item, 0);
    }
    if (threadIdx.x < 32) {
      const int lane = threadIdx.x;
      int nb = -1, ng = gen + 1;
      if (lane < 6) nb = sm.q_nb[lane];
      else if (lane == 6 && sm.active) { nb = item; ng = gen + 2; }
      bool won = false;
      if (ng < gens && nb >= 0) won = atomicExch(ts.d_flag_pr + nb, 1) == 0;
      const unsigned m = __ballot_sync(jfc::FULL, won);
      if (m && lane == 0) atomicAdd(&ctr->pr_out, __popc(m));   // counted before they can finish
      // (a failed put raises the error flag; the next dequeue sees it and
      // every thread of the CTA leaves the loop together)
      if (won) pr_ring_put(ring, cap, &ctr->pr_tail, &ctr->error, max_spins, ring_entry(nb, ng));
      __syncwarp();
      if (lane == 0) atomicSub(&ctr->pr_out, 1);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    if (visits) atomicAdd(&ctr->visits, visits);
    if (rounds) atomicAdd(&ctr->rounds, rounds);
    // "sweeps" of the phase: generations reached (the engine's schedule reads it)
    atomicMax(&ctr->sweeps_done, maxgen + 1);
  }
  // the phase clock: the last CTA to leave adds the elapsed time
  __shared__ bool s_last;
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(&ctr->bar_count, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_last) {
    ctr->bar_count = 0;
    ctr->ns_pr += jfc::global_ns() - t0;
  }
}

template <int DIMS, int TY, int TZ, bool SPLIT = false>
cudaError_t launch_t(const TileSet& ts, int sweeps, int local_iters, cudaStream_t st, int sched) {
  constexpr int NT = Tile<DIMS, TY, TZ>::NT;
  const bool async = sched == 2 && ts.d_pr_ring != nullptr;
  const void* fn = async ? (const void*)k_pr_async<DIMS, TY, TZ, SPLIT> : (const void*)k_pr_phase<DIMS, TY, TZ, SPLIT>;
  // staging buffers in dynamic shared memory: two for the sweeps (one being
  // visited, one being filled), one for the worklist; + 128 B to align them
  const size_t dyn = sizeof(PrStage<DIMS, TY, TZ>) * (async ? 1 : 2) + 128;
  static int cache_sweeps[64] = {0}, cache_async[64] = {0};
  // without this opt-in a kernel's dynamic shared memory is limited to 48 KB
  // minus its static shared memory
  {
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
    if (e != cudaSuccess) return e;
  }
  const int blocks = persistent_blocks_cached(async ? cache_async : cache_sweeps, fn, NT, dyn);
  TileSet arg = ts;
  void* params[] = {(void*)&arg, (void*)&sweeps, (void*)&local_iters};
  jfc_note_launch();
  return cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(NT), params, dyn, st);
}

// Local pre-push before the first relabel of a solve, one CTA per tile, the
// tile in shared memory: along one arc slot at a time, every node with excess
// pushes to its in-tile neighbour across that slot when the neighbour is a
// deficit, at most the arc's residual and the deficit.  Along one slot a node
// either sends (e > 0) or receives (e < 0, from its one neighbour on the other
// side), so each step is race-free; JFC_PREPUSH_ROUNDS rounds over all slots.
// These are ordinary preflow pushes (the exact relabel that follows gives
// valid heights), so the maximum flow and the canonical cut do not change;
// most of the excess that meets a deficit a step or two away cancels here, in
// one read and one write of the tile, instead of in push-relabel visits.
#ifndef JFC_PREPUSH_ROUNDS
#define JFC_PREPUSH_ROUNDS 2
#endif
template <int DIMS, int TY, int TZ>
__global__ void __launch_bounds__(Tile<DIMS, TY, TZ>::NT) k_prepush(TileSet ts) {
  using T = Tile<DIMS, TY, TZ>;
  __shared__ int se[T::NT];
  __shared__ int sr[T::K][T::NT];
  const int t = threadIdx.x;
  const int x = t & 31, row = t >> 5, y = row % TY, z = row / TY;
  const int4 ti = ts.d_info[blockIdx.x];
  const GridDev& g = ts.d_desc[ti.x];
  const long long pitch = g.pitch, slab = (long long)g.pitch * g.Hp;
  const long long n = (long long)ti.y * 32 + x + ((long long)ti.z * TY + y) * pitch + ((long long)ti.w * TZ + z) * slab;
  const int e0 = g.e[n];
  int r0[T::K];
#pragma unroll
  for (int k = 0; k < T::K; ++k) r0[k] = g.r[k][n];
  // nothing to do unless the tile holds both excess and a deficit
  const bool pos = __syncthreads_or(e0 > 0);
  const bool neg = __syncthreads_or(e0 < 0);
  if (!pos || !neg) return;
  se[t] = e0;
#pragma unroll
  for (int k = 0; k < T::K; ++k) sr[k][t] = r0[k];
  __syncthreads();
  for (int rnd = 0; rnd < JFC_PREPUSH_ROUNDS; ++rnd) {
#pragma unroll
    for (int k = 0; k < T::K; ++k) {
      const bool inside = k == T::XP ? x < 31 : k == T::XM ? x > 0 : k == T::YP ? y < TY - 1
                        : k == T::YM ? y > 0 : k == T::ZP ? z < TZ - 1 : z > 0;
      const int off = k == T::XP ? 1 : k == T::XM ? -1 : k == T::YP ? 32 : k == T::YM ? -32
                    : k == T::ZP ? 32 * TY : -32 * TY;
      const int e = se[t];
      if (inside && e > 0) {
        const int r = sr[k][t], ev = se[t + off];
        if (r > 0 && ev < 0) {
          const int d = min(min(e, r), -ev);
          se[t] = e - d;
          sr[k][t] = r - d;
          se[t + off] = ev + d;
          sr[T::K - 1 - k][t + off] += d;
        }
      }
      __syncthreads();
    }
  }
  const int e1 = se[t];
  if (e1 != e0) g.e[n] = e1;
#pragma unroll
  for (int k = 0; k < T::K; ++k) {
    const int v = sr[k][t];
    if (v != r0[k]) g.r[k][n] = v;
  }
}

template <int DIMS, int TY, int TZ>
cudaError_t prepush_t(const TileSet& ts, cudaStream_t st) {
  jfc_note_launch();
  k_prepush<DIMS, TY, TZ><<<(unsigned)ts.ntiles, Tile<DIMS, TY, TZ>::NT, 0, st>>>(ts);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_prepush(const TileSet& ts, cudaStream_t s) {
  if (ts.ntiles <= 0) return cudaSuccess;
  if (ts.dims == 2) return ts.TR == 8 ? prepush_t<2, 8, 1>(ts, s) : prepush_t<2, 16, 1>(ts, s);
  if (ts.TY == 4 && ts.TZ == 4) return prepush_t<3, 4, 4>(ts, s);
  if (ts.TY == 4 && ts.TZ == 2) return prepush_t<3, 4, 2>(ts, s);
  if (ts.TY == 16 && ts.TZ == 1) return prepush_t<3, 16, 1>(ts, s);
  if (ts.TY == 8 && ts.TZ == 2) return prepush_t<3, 8, 2>(ts, s);
  if (ts.TY == 8 && ts.TZ == 1) return prepush_t<3, 8, 1>(ts, s);
  return cudaErrorInvalidValue;
}

cudaError_t launch_pr_phase(const TileSet& ts, int sweeps, int local_iters, cudaStream_t s, int sched) {
  if (ts.dims == 2) {
    if (ts.pr_split && ts.TR == 16) return launch_t<2, 8, 1, true>(ts, sweeps, local_iters, s, sched);
    switch (ts.TR) {
      case 8: return launch_t<2, 8, 1>(ts, sweeps, local_iters, s, sched);
      case 16: return launch_t<2, 16, 1>(ts, sweeps, local_iters, s, sched);
      default: return cudaErrorInvalidValue;
    }
  }
  if (ts.TY == 4 && ts.TZ == 4) return launch_t<3, 4, 4>(ts, sweeps, local_iters, s, sched);
  if (ts.TY == 4 && ts.TZ == 2) return launch_t<3, 4, 2>(ts, sweeps, local_iters, s, sched);
  if (ts.TY == 16 && ts.TZ == 1) return launch_t<3, 16, 1>(ts, sweeps, local_iters, s, sched);
  if (ts.TY == 8 && ts.TZ == 2) return launch_t<3, 8, 2>(ts, sweeps, local_iters, s, sched);
  if (ts.TY == 8 && ts.TZ == 1) return launch_t<3, 8, 1>(ts, sweeps, local_iters, s, sched);
  return cudaErrorInvalidValue;
}
