// kernels_build.cu — capacity build: contrast n-links, k-means colour models,
// net-excess t-links, warm seed edits.
//
// Reference: graphcut_compute_capacity_bk/_lazy (graphcut_compute_capacity.cl:21-254),
// graphcut_kmeans (graphcut_kmeans.cl:21-159) with the host loop
// QGCWidget::kmeans (QGCWidget.cpp:1997-2107) moved onto the device,
// graphcut_compute_excessflow_lazy (graphcut_compute_excessflow.cl:47-77, 109-139).
// The reference evaluates exp / log in float on the device; here every
// floating-point step happens once on the host in double into int32 lookup
// tables (n-link weight per contrast index, t-link cost per quantised
// probability), and the device only does integer arithmetic and table
// gathers, so the device build is bit-identical to the CPU restatement.
//   n-link  w = LUT[|dI|] (scalar) or LUT[||dI||^2] (RGB), symmetric
//   model   fixed-point (1/16) k-means over seed pixels, integer distances
//   t-link  q = floor(Q dF / (dF + dB)); cs = LUTs[q], ct = LUTt[q];
//           seeds: cs / ct = seed_cap; e = cs - ct; sink_total += ct
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "jfc_internal.h"

namespace cg = cooperative_groups;

namespace {

constexpr unsigned FULL = 0xffffffffu;

template <int PF>
__device__ __forceinline__ void feat(const void* __restrict__ img, long long i, int* f) {
  if constexpr (PF == JFC_PIX_GRAY8) {
    f[0] = ((const uint8_t*)img)[i];
  } else if constexpr (PF == JFC_PIX_RGB8) {
    const uint8_t* p = (const uint8_t*)img + 3 * i;
    f[0] = p[0]; f[1] = p[1]; f[2] = p[2];
  } else {
    f[0] = (int)((const int16_t*)img)[i] + 32768;
  }
}

template <int PF>
__device__ __forceinline__ unsigned pack_feat(const int* f) {
  if constexpr (PF == JFC_PIX_RGB8) return (unsigned)f[0] | ((unsigned)f[1] << 8) | ((unsigned)f[2] << 16);
  else return (unsigned)f[0];
}

// contrast-table index and squared difference of a neighbour pair
template <int PF>
__device__ __forceinline__ int contrast_index(const int* a, const int* b) {
  if constexpr (PF == JFC_PIX_RGB8) {
    const int d0 = a[0] - b[0], d1 = a[1] - b[1], d2 = a[2] - b[2];
    return d0 * d0 + d1 * d1 + d2 * d2;
  } else {
    const int d = a[0] - b[0];
    return d < 0 ? -d : d;
  }
}
template <int PF>
__device__ __forceinline__ unsigned contrast_sq(const int* a, const int* b) {   // (65535^2 fits 32 bits unsigned)
  const unsigned d = (unsigned)contrast_index<PF>(a, b);
  if constexpr (PF == JFC_PIX_RGB8) return d;
  else return d * d;
}

__device__ __forceinline__ void dense_xyz(const GridDev& g, long long i, int& x, int& y, int& z) {
  x = (int)(i % g.W);
  const long long yz = i / g.W;
  y = (int)(yz % g.H);
  z = (int)(yz / g.H);
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}

// Sum, over one block, of a per-thread u64; thread 0 adds it to *dst.
__device__ __forceinline__ void block_sum_to(unsigned long long v, unsigned long long* dst) {
  __shared__ unsigned long long s_part[32];
  v = warp_sum_u64(v);
  if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s_part[w];
    if (t) atomicAdd(dst, t);
  }
}

// Sum over i in [0, n - off) of (v[i] - v[i + off])^2, v the image's values
// (bytes or int16) in memory order, as this thread's share of the grid.  Pairs at
// one distance need no pixel arithmetic: 16 bytes a thread and step, the
// partner's bytes from the aligned words around them by funnel shifts, four
// byte differences and their squares in two instructions.
template <typename V>
__device__ __forceinline__ unsigned long long pair_sum(const V* __restrict__ v, long long n, long long off) {
  constexpr int E = 16 / (int)sizeof(V);   // values a step
  const long long pairs = n - off;
  const unsigned* words = reinterpret_cast<const unsigned*>(v);
  const long long wo = off * (long long)sizeof(V) / 4;
  const unsigned sh = 8u * (unsigned)(off * (long long)sizeof(V) & 3);
  unsigned long long acc = 0;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c * E < pairs;
       c += (long long)gridDim.x * blockDim.x) {
    const long long i = c * E;
    if (i + E + off + 4 / (long long)sizeof(V) <= n) {
      const uint4 a4 = *reinterpret_cast<const uint4*>(words + 4 * c);
      const unsigned a[4] = {a4.x, a4.y, a4.z, a4.w};
      unsigned b[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) b[k] = words[4 * c + wo + k];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const unsigned p = __funnelshift_r(b[k], b[k + 1], sh);
        if constexpr (sizeof(V) == 1) {
          const unsigned d = __vabsdiffu4(a[k], p);
          acc += (unsigned long long)__dp4a(d, d, 0u);
        } else {
          const unsigned d = __vabsdiffs2(a[k], p);
          acc += (unsigned long long)(d & 0xffffu) * (d & 0xffffu) + (unsigned long long)(d >> 16) * (d >> 16);
        }
      }
    } else {
      for (long long j = i; j < i + E && j < pairs; ++j) {
        const long long d = (long long)v[j] - v[j + off];
        acc += (unsigned long long)(d * d);
      }
    }
  }
  return acc;
}

// Sum of squared neighbour differences over every +x / +y (/ +z) pair: all pairs
// of values one pixel, one row (and one slice) apart in memory, less those that
// join the end of a row or slice to the start of the next (sums are modulo
// 2^64, the result is their true value).  Pixel by pixel with its neighbours
// loaded as bytes it took 506 us on 15000 x 10000 RGB and 33 us on 1920 x 1080;
// this 240 and 7 (70 at the HBM rate).
template <int PF, int DIMS>
__global__ void __launch_bounds__(256) k_contrast_sum(GridDev g, const void* __restrict__ img,
                                                      unsigned long long* sum) {
  using V = typename std::conditional<PF == JFC_PIX_I16, int16_t, uint8_t>::type;
  constexpr int C = PF == JFC_PIX_RGB8 ? 3 : 1;
  const V* v = (const V*)img;
  const long long W = (long long)g.W * C, rows = (long long)g.H * g.D, n = W * rows, slab = W * g.H;
  unsigned long long acc = pair_sum<V>(v, n, C) + pair_sum<V>(v, n, W);
  if (DIMS == 3) acc += pair_sum<V>(v, n, slab);
  const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, tn = (long long)gridDim.x * blockDim.x;
  auto less = [&](long long i, long long j) {
    const long long d = (long long)v[i] - v[j];
    acc -= (unsigned long long)(d * d);
  };
  for (long long r = t0; r + 1 < rows; r += tn)   // row r's last pixel and row r + 1's first
    for (int c = 0; c < C; ++c) less((r + 1) * W - C + c, (r + 1) * W + c);
  if (DIMS == 3)
    for (long long i = t0; i < W * (g.D - 1); i += tn) {   // slice z's last row and slice z + 1's first
      const long long j = (i / W + 1) * slab + i % W;
      less(j - W, j);
    }
  block_sum_to(acc, sum);
}

// Seed statistics per class: count, per-channel min / max, and (fill) the
// packed features of the seed pixels (order is irrelevant: the k-means below
// is order-free).  Each thread takes 16 seed bytes at a time with one vector
// load and skips them when all are unseeded (the common case); list slots
// are reserved once per warp from per-thread class counts.
__device__ __forceinline__ int count_bytes_eq(const uint4& v, unsigned pat) {
  return (__popc(__vcmpeq4(v.x, pat)) + __popc(__vcmpeq4(v.y, pat)) + __popc(__vcmpeq4(v.z, pat)) +
          __popc(__vcmpeq4(v.w, pat))) >> 3;
}

template <int PF>
__global__ void __launch_bounds__(256) k_seed_stats(GridDev g, const void* __restrict__ img,
                                                    const uint8_t* __restrict__ seeds, int* minmax,
                                                    unsigned long long* count, uint32_t* list_f,
                                                    uint32_t* list_b, unsigned int* fill, int do_fill) {
  __shared__ int s_mm[2][3][2];
  __shared__ unsigned long long s_cnt[2];
  if (threadIdx.x < 12) ((int*)s_mm)[threadIdx.x] = (threadIdx.x & 1) ? -1 : 0x7fffffff;
  if (threadIdx.x < 2) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  constexpr int C = PF == JFC_PIX_RGB8 ? 3 : 1;
  const long long n = (long long)g.W * g.H * g.D;
  const long long chunks = (n + 15) / 16;
  const int lane = threadIdx.x & 31;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long start = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long iters = (chunks + stride - 1) / stride;
  int mn[2][C], mx[2][C];
  for (int k = 0; k < 2; ++k)
    for (int c = 0; c < C; ++c) { mn[k][c] = 0x7fffffff; mx[k][c] = -1; }
  unsigned long long cnt[2] = {0, 0};
  for (long long it = 0; it < iters; ++it) {
    const long long ch = start + it * stride;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (ch < chunks) {
      const long long i0 = ch * 16;
      if (i0 + 16 <= n) {
        v = __ldg(reinterpret_cast<const uint4*>(seeds + i0));
      } else {
        unsigned long long lo = 0, hi = 0;
        for (int b = 0; b < 16 && i0 + b < n; ++b) {
          const unsigned long long t = (unsigned long long)seeds[i0 + b];
          if (b < 8) lo |= t << (8 * b);
          else hi |= t << (8 * (b - 8));
        }
        v = make_uint4((unsigned)lo, (unsigned)(lo >> 32), (unsigned)hi, (unsigned)(hi >> 32));
      }
    }
    const bool any = (v.x | v.y | v.z | v.w) != 0;
    if (!__any_sync(FULL, any)) continue;
    const int c1 = any ? count_bytes_eq(v, 0x01010101u) : 0;
    const int c2 = any ? count_bytes_eq(v, 0x02020202u) : 0;
    cnt[0] += c1;
    cnt[1] += c2;
    unsigned pos1 = 0, pos2 = 0;
    if (do_fill) {
      // exclusive warp scans of the per-thread counts, one reservation per class
      unsigned s1 = c1, s2 = c2;
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned t1 = __shfl_up_sync(FULL, s1, o), t2 = __shfl_up_sync(FULL, s2, o);
        if (lane >= o) { s1 += t1; s2 += t2; }
      }
      unsigned b1 = 0, b2 = 0;
      if (lane == 31) {
        if (s1) b1 = atomicAdd(&fill[0], s1);
        if (s2) b2 = atomicAdd(&fill[1], s2);
      }
      b1 = __shfl_sync(FULL, b1, 31);
      b2 = __shfl_sync(FULL, b2, 31);
      pos1 = b1 + s1 - c1;
      pos2 = b2 + s2 - c2;
    }
    if (!any) continue;
#pragma unroll
    for (int b = 0; b < 16; ++b) {
      const unsigned w = b < 4 ? v.x : b < 8 ? v.y : b < 12 ? v.z : v.w;
      const int sd = (w >> (8 * (b & 3))) & 255;
      if (sd != 1 && sd != 2) continue;
      int f[3] = {0, 0, 0};
      feat<PF>(img, ch * 16 + b, f);
      if (sd == 1) {
#pragma unroll
        for (int c = 0; c < C; ++c) { mn[0][c] = min(mn[0][c], f[c]); mx[0][c] = max(mx[0][c], f[c]); }
        if (do_fill) list_f[pos1++] = pack_feat<PF>(f);
      } else {
#pragma unroll
        for (int c = 0; c < C; ++c) { mn[1][c] = min(mn[1][c], f[c]); mx[1][c] = max(mx[1][c], f[c]); }
        if (do_fill) list_b[pos2++] = pack_feat<PF>(f);
      }
    }
  }
  for (int k = 0; k < 2; ++k)
    for (int c = 0; c < C; ++c) {
      const int lo = __reduce_min_sync(FULL, mn[k][c]), hi = __reduce_max_sync(FULL, mx[k][c]);
      if (lane == 0) {
        if (lo != 0x7fffffff) atomicMin(&s_mm[k][c][0], lo);
        if (hi >= 0) atomicMax(&s_mm[k][c][1], hi);
      }
    }
  for (int k = 0; k < 2; ++k) {
    const unsigned long long t = warp_sum_u64(cnt[k]);
    if (lane == 0 && t) atomicAdd(&s_cnt[k], t);
  }
  __syncthreads();
  if (threadIdx.x < 12) {
    const int v = ((int*)s_mm)[threadIdx.x];
    if (threadIdx.x & 1) { if (v >= 0) atomicMax(&minmax[threadIdx.x], v); }
    else if (v != 0x7fffffff) atomicMin(&minmax[threadIdx.x], v);
  }
  if (threadIdx.x < 2 && s_cnt[threadIdx.x]) atomicAdd(&count[threadIdx.x], s_cnt[threadIdx.x]);
}

__device__ __forceinline__ void unpack_feat(unsigned v, int C, int* f) {
  if (C == 3) { f[0] = v & 255; f[1] = (v >> 8) & 255; f[2] = (v >> 16) & 255; }
  else f[0] = (int)v;
}

// Squared distance of a feature (scaled by 16) to a fixed-point centre.  For
// 8-bit features every term is below 2^24 and the sum below 2^26, so 32-bit
// arithmetic is exact; 16-bit features need 64 bits.
template <int PF> struct Dist { using T = int; };
template <> struct Dist<JFC_PIX_I16> { using T = long long; };

template <int PF>
__device__ __forceinline__ typename Dist<PF>::T fdist(const int* f, const int* mu) {
  using T = typename Dist<PF>::T;
  constexpr int C = PF == JFC_PIX_RGB8 ? 3 : 1;
  T s = 0;
  for (int c = 0; c < C; ++c) {
    const T t = (T)16 * f[c] - mu[c];
    s += t * t;
  }
  return s;
}

// Sum of each of NV (32 or 16) per-lane values over the warp by a transposing
// butterfly, NV - 1 (+ NV) shuffles instead of 5 NV: lane l returns value l % NV.
template <int NV, typename T>
__device__ __forceinline__ T warp_transpose_sum(T (&v)[NV]) {
  const int lane = threadIdx.x & 31;
  if constexpr (NV == 16) {
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] += __shfl_xor_sync(FULL, v[i], 16);
  }
#pragma unroll
  for (int w = NV / 2; w; w >>= 1) {
    const bool up = (lane & w) != 0;
#pragma unroll
    for (int i = 0; i < w; ++i) {
      const T keep = up ? v[i + w] : v[i], send = up ? v[i] : v[i + w];
      v[i] = keep + __shfl_xor_sync(FULL, send, w);
    }
  }
  return v[0];
}

// k-means over both classes' seed lists: all iterations in one launch, until
// no class moves or `iters` ran.  Every block keeps its own copy of the
// centres and updates it from the same totals (rounded mean, fixed point 1/16,
// integer sums, so the order of the sums does not matter).  Up to 8 centres a
// class are summed in registers, more by shared-memory atomics.
// CLUSTER: the blocks are one cluster and read each other's sums through
// distributed shared memory, one cluster barrier an iteration; else the sums go
// through global memory behind a grid barrier (cooperative launch; three
// buffers: the one after next is cleared while the current one is summed).
// One launch per iteration, the last block moving the centres, took 9-13 us an
// iteration at any list length below 20,000 and 2 us for each iteration left
// over after convergence: 105 us for the 499 seeds of a 640 x 480 image, 219
// us for 10,282 and 517 us for 880,711 seeds of RGB images, against 20, 101 and
// 244 us here.
constexpr int kKmThreads = 1024;
constexpr unsigned long long kKmPolls = 1ull << 26;   // grid barrier: polls before it gives up
template <int PF, bool CLUSTER>
__global__ void __launch_bounds__(kKmThreads, 1) k_kmeans(const uint32_t* __restrict__ list, KmeansDev* km, int iters) {
  constexpr int C = PF == JFC_PIX_RGB8 ? 3 : 1;
  constexpr int KR = 8, NV = (C + 1) * KR;   // register sums: channel-major, counts last
  using T = typename Dist<PF>::T;
  using S = typename std::conditional<PF == JFC_PIX_I16, unsigned long long, unsigned>::type;
  __shared__ int s_mu[2][JFC_MAX_K * 3];
  __shared__ unsigned long long s_acc[2][2][JFC_MAX_K * 4];   // [iteration & 1][class][centre * 4 + channel or count]
  __shared__ unsigned long long s_tot[2][JFC_MAX_K * 4];
  __shared__ int s_moved[2], s_ok;
  const int t = threadIdx.x, lane = t & 31;
  const long long stride = (long long)gridDim.x * kKmThreads, start = (long long)blockIdx.x * kKmThreads + t;
  for (int i = t; i < 2 * JFC_MAX_K * 3; i += kKmThreads) (&s_mu[0][0])[i] = (&km->mu[0][0])[i];
  bool live[2] = {true, true};   // the class still moves
  bool ok = true;
  for (int it = 0; it < iters && ok && (live[0] || live[1]); ++it) {
    unsigned long long(*acc)[JFC_MAX_K * 4] = s_acc[it & 1];
    for (int i = t; i < 2 * JFC_MAX_K * 4; i += kKmThreads) (&acc[0][0])[i] = 0;
    if (t < 2) s_moved[t] = 0;
    __syncthreads();
    for (int cls = 0; cls < 2; ++cls) {
      if (!live[cls]) continue;
      const int k = km->k[cls];
      const long long n = (long long)km->n[cls];
      const uint32_t* L = list + (cls ? km->n[0] : 0ull);
      const int* mu = s_mu[cls];
      auto nearest = [&](const int* f) {
        int best = 0;
        T bd = fdist<PF>(f, mu);
        for (int j = 1; j < k; ++j) {
          const T d = fdist<PF>(f, mu + 3 * j);
          if (d < bd) { bd = d; best = j; }
        }
        return best;
      };
      if (k <= KR) {
        unsigned v[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) v[i] = 0;
        for (long long i = start; i < n; i += stride) {
          int f[3] = {0, 0, 0};
          unpack_feat(L[i], C, f);
          const int best = nearest(f);
#pragma unroll
          for (int j = 0; j < KR; ++j) {
            const bool m = best == j;
#pragma unroll
            for (int c = 0; c < C; ++c) v[c * KR + j] += m ? (unsigned)f[c] : 0u;
            v[C * KR + j] += m ? 1u : 0u;
          }
        }
        S w[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) w[i] = v[i];
        const S sum = warp_transpose_sum<NV, S>(w);
        // value c * KR + j -> slot j * 4 + c (counts: slot j * 4 + 3)
        const int c = lane / KR, j = lane % KR;
        if (lane < NV && sum) atomicAdd(&acc[cls][j * 4 + (c == C ? 3 : c)], (unsigned long long)sum);
      } else {
        for (long long i = start; i < n; i += stride) {
          int f[3] = {0, 0, 0};
          unpack_feat(L[i], C, f);
          const int best = nearest(f);
#pragma unroll
          for (int c = 0; c < C; ++c) atomicAdd(&acc[cls][best * 4 + c], (unsigned long long)f[c]);
          atomicAdd(&acc[cls][best * 4 + 3], 1ull);
        }
      }
    }
    const int cls = t / (JFC_MAX_K * 4), slot = t % (JFC_MAX_K * 4);   // (t < 256)
    if constexpr (CLUSTER) {
      cg::cluster_group cl = cg::this_cluster();
      cl.sync();
      if (t < 2 * JFC_MAX_K * 4) {
        unsigned long long v = 0;
        for (unsigned r = 0; r < cl.num_blocks(); ++r) v += cl.map_shared_rank(&acc[cls][slot], r)[0];
        s_tot[cls][slot] = v;
      }
    } else {
      __syncthreads();
      if (t < 2 * JFC_MAX_K * 4) {
        if (acc[cls][slot]) atomicAdd(&km->acc[it % 3][cls][slot], acc[cls][slot]);
        if (blockIdx.x == 0) km->acc[(it + 1) % 3][cls][slot] = 0;   // last read two iterations ago
      }
      __syncthreads();
      if (t == 0) {
        __threadfence();
        atomicAdd(&km->bar, 1ull);
        const unsigned long long target = (unsigned long long)(it + 1) * gridDim.x;
        unsigned long long spins = 0;
        int good = 1;
        while (*(volatile unsigned long long*)&km->bar < target) {
          if (*(volatile int*)&km->error || ++spins > kKmPolls) {
            atomicExch(&km->error, 1);
            good = 0;
            break;
          }
          if (spins > 16) __nanosleep(40);
        }
        __threadfence();
        s_ok = good;
      }
      __syncthreads();
      ok = s_ok != 0;
      if (t < 2 * JFC_MAX_K * 4) s_tot[cls][slot] = __ldcg(&km->acc[it % 3][cls][slot]);
    }
    __syncthreads();
    if (ok && t < 2 * JFC_MAX_K * 3) {
      const int q = t / (JFC_MAX_K * 3), r = t % (JFC_MAX_K * 3), j = r / 3, c = r % 3;
      if (live[q] && j < km->k[q] && c < C) {
        const long long c4 = (long long)s_tot[q][j * 4 + 3];
        if (c4 != 0) {
          const int v = (int)((16 * (long long)s_tot[q][j * 4 + c] + c4 / 2) / c4);
          if (v != s_mu[q][r]) {
            s_mu[q][r] = v;
            s_moved[q] = 1;
          }
        }
      }
    }
    __syncthreads();
    for (int q = 0; q < 2; ++q) live[q] = live[q] && s_moved[q] != 0;
    __syncthreads();   // (s_moved is cleared by the next iteration)
  }
  if constexpr (CLUSTER) cg::this_cluster().sync();   // (no block leaves while another reads its sums)
  if (blockIdx.x == 0)
    for (int i = t; i < 2 * JFC_MAX_K * 3; i += kKmThreads) (&km->mu[0][0])[i] = (&s_mu[0][0])[i];
}

// Colour models as the t-link pass reads them, in shared memory: for centre mu
// the squared distance of a feature f (scaled by 16) is |16 f|^2 + (|mu|^2 -
// 32 f.mu), so a centre costs one multiply-add per channel and a minimum.
template <int PF>
struct TlinkModel {
  static constexpr int C = PF == JFC_PIX_RGB8 ? 3 : 1;
  using T = typename Dist<PF>::T;
  struct alignas(16) Centre {
    T sq;        // |mu|^2
    int m[3];    // -32 mu
  };
  Centre c[2][JFC_MAX_K];
  int k[2];
};

// Fill the block's model (all threads call it; a barrier follows).
template <int PF>
__device__ __forceinline__ void load_model(TlinkModel<PF>& s, const BuildModelDev& m, const int* __restrict__ mu) {
  constexpr int C = TlinkModel<PF>::C;
  for (int i = threadIdx.x; i < 2 * JFC_MAX_K; i += blockDim.x) {
    const int cls = i / JFC_MAX_K, j = i % JFC_MAX_K;
    typename TlinkModel<PF>::Centre c;
    c.sq = 0;
    for (int ch = 0; ch < 3; ++ch) {
      const int v = ch < C ? mu[cls * JFC_MAX_K * 3 + 3 * j + ch] : 0;
      c.sq += (typename TlinkModel<PF>::T)v * v;
      c.m[ch] = -32 * v;
    }
    s.c[cls][j] = c;
  }
  if (threadIdx.x == 0) {
    s.k[0] = m.kf;
    s.k[1] = m.kb;
  }
}

// min over the centres of |mu|^2 - 32 f.mu for N nodes; unrolled for up to 8
// centres (a loop of one centre is as much branch as arithmetic).
template <int PF, int K, int N>
__device__ __forceinline__ void nearest_of(const typename TlinkModel<PF>::Centre* s, const int (&f)[N][3],
                                           typename Dist<PF>::T (&best)[N], bool more = false) {
  using T = typename Dist<PF>::T;
#pragma unroll
  for (int j = 0; j < K; ++j) {
    const typename TlinkModel<PF>::Centre ce = s[j];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      T v = ce.sq;
#pragma unroll
      for (int c = 0; c < TlinkModel<PF>::C; ++c) v += (T)f[i][c] * ce.m[c];
      best[i] = j == 0 && !more ? v : min(best[i], v);
    }
  }
}
template <int PF, int N>
__device__ __forceinline__ void nearest_centre(const typename TlinkModel<PF>::Centre* s, int k, const int (&f)[N][3],
                                               typename Dist<PF>::T (&best)[N]) {
  switch (k) {
    case 1: nearest_of<PF, 1, N>(s, f, best); return;
    case 2: nearest_of<PF, 2, N>(s, f, best); return;
    case 3: nearest_of<PF, 3, N>(s, f, best); return;
    case 4: nearest_of<PF, 4, N>(s, f, best); return;
    case 5: nearest_of<PF, 5, N>(s, f, best); return;
    case 6: nearest_of<PF, 6, N>(s, f, best); return;
    case 7: nearest_of<PF, 7, N>(s, f, best); return;
    default: break;
  }
  nearest_of<PF, 8, N>(s, f, best);
  for (int j = 8; j < k; ++j) nearest_of<PF, 1, N>(s + j, f, best, true);
}

// t-link costs of N nodes.  q = floor(Q dF / (dF + dB)): a float quotient lands
// within 1 of q (its relative error is below 2^-21, q below 2^16) and one exact
// integer step either way corrects it (8-bit features: dF + dB < 2^27; 16-bit:
// < 2^42, the products below 2^59).
// (tab: cost of the source link at q; the sink link's is the same table's at
// the complementary probability, JFC_TQ - q)
template <int PF, int N, typename Tab>
__device__ __forceinline__ void tlinks(const TlinkModel<PF>& s, int seed_cap, const Tab* __restrict__ tab,
                                       const int (&f)[N][3], const int (&seed)[N], int (&cs)[N], int (&ct)[N]) {
  constexpr int C = TlinkModel<PF>::C;
  using T = typename Dist<PF>::T;
  using U = typename std::conditional<PF == JFC_PIX_I16, unsigned long long, unsigned>::type;
  T dF[N], dB[N];
  nearest_centre<PF, N>(s.c[0], s.k[0], f, dF);
  nearest_centre<PF, N>(s.c[1], s.k[1], f, dB);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    T ff = 0;
#pragma unroll
    for (int c = 0; c < C; ++c) ff += (T)(16 * f[i][c]) * (16 * f[i][c]);
    const U d = (U)(dF[i] + ff), sum = d + (U)(dB[i] + ff);
    unsigned q = JFC_TQ / 2;
    if (sum != 0) {
      q = (unsigned)(__fdividef((float)d, (float)sum) * (float)JFC_TQ);
      const unsigned long long num = (unsigned long long)JFC_TQ * d, qs = (unsigned long long)q * sum;
      if (qs > num) --q;
      else if (qs + sum <= num) ++q;
    }
    cs[i] = tab[q];
    ct[i] = tab[JFC_TQ - q];
    if (seed[i] == JFC_SEED_FG) { cs[i] = seed_cap; ct[i] = 0; }
    if (seed[i] == JFC_SEED_BG) { cs[i] = 0; ct[i] = seed_cap; }
  }
}

// Table entry t takes the value of the last run that starts at or before it
// (a bisection of the few hundred starts, which stay in L1), as an int and / or
// as a byte.
__global__ void __launch_bounds__(256) k_expand_runs(const int* __restrict__ start, const int* __restrict__ val, int m,
                                                     int n, int* __restrict__ out, uint8_t* __restrict__ out8) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  int lo = 0, hi = m;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (start[mid] <= t) lo = mid;
    else hi = mid;
  }
  const int v = val[lo];
  if (out) out[t] = v;
  if (out8) out8[t] = (uint8_t)v;
}

// Features of 4 neighbouring pixels from pixel i on, one word each (RGB: bytes
// r, g, b, 0; 16 bits: value + 32768), by aligned word loads and funnel shifts;
// total: pixels of the image (what the words would reach past its end is not
// read).
template <int PF>
__device__ __forceinline__ void feat4(const void* __restrict__ img, long long i, long long total, unsigned (&f)[4]) {
  constexpr int B = PF == JFC_PIX_RGB8 ? 3 : PF == JFC_PIX_I16 ? 2 : 1;   // bytes a pixel = words of 4 pixels
  const long long at = i * B;
  if (at + 4 * B + 4 <= total * B) {
    const unsigned* w = reinterpret_cast<const unsigned*>(img) + (at >> 2);
    const unsigned sh = 8u * (unsigned)(at & 3);
    unsigned v[B + 1], u[B];
#pragma unroll
    for (int k = 0; k <= B; ++k) v[k] = w[k];
#pragma unroll
    for (int k = 0; k < B; ++k) u[k] = __funnelshift_r(v[k], v[k + 1], sh);
    if constexpr (PF == JFC_PIX_RGB8) {
      f[0] = u[0] & 0xffffffu;
      f[1] = __funnelshift_r(u[0], u[1], 24) & 0xffffffu;
      f[2] = __funnelshift_r(u[1], u[2], 16) & 0xffffffu;
      f[3] = u[2] >> 8;
    } else if constexpr (PF == JFC_PIX_I16) {
#pragma unroll
      for (int k = 0; k < 4; ++k) f[k] = ((u[k / 2] >> (16 * (k & 1))) & 0xffffu) ^ 0x8000u;
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) f[k] = (u[0] >> (8 * k)) & 255u;
    }
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      int a[3] = {0, 0, 0};
      if (i + k < total) feat<PF>(img, i + k, a);
      f[k] = i + k < total ? pack_feat<PF>(a) : 0u;
    }
  }
}

// contrast-table index of two packed features
template <int PF>
__device__ __forceinline__ int contrast4(unsigned a, unsigned b) {
  if constexpr (PF == JFC_PIX_RGB8) {
    const unsigned d = __vabsdiffu4(a, b);
    return (int)__dp4a(d, d, 0u);
  } else {
    return a > b ? (int)(a - b) : (int)(b - a);
  }
}

// One pass over the padded grid: n-links (both directions of every pair, from
// the contrast table), t-links, e = cs - ct, label = 0; padding is zeroed.
// A lane takes 4 neighbouring columns and walks down `rows` rows: pixels come as
// words, planes leave as 128-bit stores, a centre is read once for 4 nodes, the
// weight to the right is the next node's weight to the left, the weight down
// the next row's weight up (across the ends of a strip they are computed
// again; along z both are, each slice on its own).
// BYTES: every weight and cost fits a byte (default scales: 100 and 118), so the
// block holds the tables in shared memory (32 lanes' look-ups in tables of
// 256-780 KB are up to 32 accesses of L1 each).
// With a node a lane the pass was bound by instructions, 320 per 32 nodes:
// 2.03 ms on 15000 x 10000 RGB (0.67 at the HBM rate) and, with a 64-bit division
// per node, 0.40 ms on 317 x 301 x 181 int16; this 1.24 and 0.25 (60% of the
// issue slots).
struct BuildTables {
  const int* xy;         // n-link weights over the contrast index (int), used when !BYTES
  const int* z;
  const int* t;          // t-link costs over the quantised probability
  const uint8_t* xy8;    // the same as bytes (padded to 16): entries past the last are the last
  const uint8_t* z8;
  const uint8_t* t8;
  int nxy, nz;           // entries of xy8, z8
};
constexpr int kBuildThreads = 384;
__host__ __device__ constexpr int pad16(int v) { return (v + 15) / 16 * 16; }
template <int PF, int DIMS, bool BYTES>
__global__ void __launch_bounds__(kBuildThreads, 2) k_build(GridDev g, const void* __restrict__ img,
                                                            const uint8_t* __restrict__ seeds, BuildModelDev m,
                                                            const int* __restrict__ mu, BuildTables tb, int rows,
                                                            unsigned long long* sink) {
  __shared__ TlinkModel<PF> s_m;
  extern __shared__ __align__(16) uint8_t s_tab[];   // t8, xy8, z8
  load_model<PF>(s_m, m, mu);
  uint8_t* const s_xy = s_tab + pad16(JFC_TQ + 1);
  uint8_t* const s_z = s_xy + pad16(tb.nxy);
  if constexpr (BYTES) {
    auto copy = [](uint8_t* d, const uint8_t* src, int n) {
      for (int i = threadIdx.x; i < n / 16; i += kBuildThreads)
        reinterpret_cast<uint4*>(d)[i] = reinterpret_cast<const uint4*>(src)[i];
    };
    copy(s_tab, tb.t8, pad16(JFC_TQ + 1));
    copy(s_xy, tb.xy8, pad16(tb.nxy));
    if (DIMS == 3) copy(s_z, tb.z8, pad16(tb.nz));
  }
  __syncthreads();
  auto w_xy = [&](unsigned a, unsigned b) -> int {
    const int d = contrast4<PF>(a, b);
    if constexpr (BYTES) return s_xy[min(d, tb.nxy - 1)];
    else return tb.xy[d];
  };
  auto w_z = [&](unsigned a, unsigned b) -> int {
    const int d = contrast4<PF>(a, b);
    if constexpr (BYTES) return s_z[min(d, tb.nz - 1)];
    else return tb.z[d];
  };
  const int lane = threadIdx.x & 31;
  const int cols = (g.pitch + 127) / 128, bands = (g.Hp + rows - 1) / rows;
  const long long items = (long long)cols * bands * g.Dp, wh = (long long)g.W * g.H, total = wh * g.D;
  const int warps = kBuildThreads / 32 * gridDim.x;
  unsigned long long acc = 0;
  for (long long it = blockIdx.x * (kBuildThreads / 32) + (threadIdx.x >> 5); it < items; it += warps) {
    const int bx = (int)(it % cols);
    const long long yz = it / cols;
    const int y0 = (int)(yz % bands) * rows, z = (int)(yz / bands);
    const int x = bx * 128 + 4 * lane, y1 = min(y0 + rows, g.Hp);
    const bool store = x < g.pitch;
    const bool col = x < g.W && z < g.D;                // the first of the 4 columns is real
    const int nreal = col ? min(4, g.W - x) : 0;        // real columns
    long long i = (long long)z * wh + (long long)y0 * g.W + x;
    long long p = (long long)x + (long long)g.pitch * (y0 + (long long)g.Hp * z);
    unsigned a[4] = {0, 0, 0, 0}, n[4] = {0, 0, 0, 0};   // this row's pixels, the next row's
    int w_ym[4] = {0, 0, 0, 0};
    if (col && y0 < g.H) {
      feat4<PF>(img, i, total, a);
      if (y0 > 0) {
        feat4<PF>(img, i - g.W, total, n);
#pragma unroll
        for (int k = 0; k < 4; ++k) w_ym[k] = k < nreal ? w_xy(a[k], n[k]) : 0;
      }
    }
    for (int y = y0; y < y1; ++y, i += g.W, p += g.pitch) {
      const bool real = col && y < g.H, below = col && y + 1 < g.H;
      if (below) feat4<PF>(img, i + g.W, total, n);
      // seeds: one by one (rows start at any byte)
      int seed[4] = {0, 0, 0, 0};
      if (real) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (k < nreal) seed[k] = seeds[i + k];
      }
      // the pixel beside the warp's strip: lane 31 to the right, lane 0 to the left
      unsigned beside = 0;
      const bool has = real && ((lane == 31 && x + 4 < g.W) || (lane == 0 && x > 0));
      if (has) {
        int e[3] = {0, 0, 0};
        feat<PF>(img, lane == 0 ? i - 1 : i + 4, e);
        beside = pack_feat<PF>(e);
      }
      unsigned right = __shfl_down_sync(FULL, a[0], 1);
      if (lane == 31) right = beside;
      int w_xp[4], w_xm[4], w_yp[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        w_xp[k] = real && x + k + 1 < g.W ? w_xy(a[k], k < 3 ? a[k < 3 ? k + 1 : 3] : right) : 0;
        w_yp[k] = below && k < nreal ? w_xy(a[k], n[k]) : 0;
      }
      w_xm[0] = __shfl_up_sync(FULL, w_xp[3], 1);
      if (lane == 0) w_xm[0] = has ? w_xy(a[0], beside) : 0;
      if (!real) w_xm[0] = 0;
#pragma unroll
      for (int k = 1; k < 4; ++k) w_xm[k] = w_xp[k - 1];
      int cs[4] = {0, 0, 0, 0}, ct[4] = {0, 0, 0, 0};
      if (real) {
        int f[4][3];
#pragma unroll
        for (int k = 0; k < 4; ++k) unpack_feat(a[k], PF == JFC_PIX_RGB8 ? 3 : 1, f[k]);
        if constexpr (BYTES) tlinks<PF, 4>(s_m, m.seed_cap, s_tab, f, seed, cs, ct);
        else tlinks<PF, 4>(s_m, m.seed_cap, tb.t, f, seed, cs, ct);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (!real || k >= nreal) cs[k] = ct[k] = 0;
        acc += (unsigned long long)ct[k];
      }
      if (store) {
        auto put = [&](int* plane, const int (&v)[4]) {
          *reinterpret_cast<int4*>(plane + p) = make_int4(v[0], v[1], v[2], v[3]);
        };
        put(g.r[0], w_xp);
        put(g.r[1], w_yp);
        if constexpr (DIMS == 3) {
          int w_zp[4] = {0, 0, 0, 0}, w_zm[4] = {0, 0, 0, 0};
          unsigned b[4];
          if (real && z + 1 < g.D) {
            feat4<PF>(img, i + wh, total, b);
#pragma unroll
            for (int k = 0; k < 4; ++k) w_zp[k] = k < nreal ? w_z(a[k], b[k]) : 0;
          }
          if (real && z > 0) {
            feat4<PF>(img, i - wh, total, b);
#pragma unroll
            for (int k = 0; k < 4; ++k) w_zm[k] = k < nreal ? w_z(a[k], b[k]) : 0;
          }
          put(g.r[2], w_zp);
          put(g.r[3], w_zm);
        }
        if (!real) w_ym[0] = w_ym[1] = w_ym[2] = w_ym[3] = 0;
        put(g.r[DIMS == 3 ? 4 : 2], w_ym);
        put(g.r[DIMS == 3 ? 5 : 3], w_xm);
        const int e[4] = {cs[0] - ct[0], cs[1] - ct[1], cs[2] - ct[2], cs[3] - ct[3]};
        put(g.e, e);
        *reinterpret_cast<unsigned*>(g.label + p) = 0u;
        if (!real || nreal < 4) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (!real || k >= nreal) g.h[p + k] = JFC_INF;
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        w_ym[k] = w_yp[k];
        a[k] = n[k];
      }
    }
  }
  block_sum_to(acc, sink);
}

// Warm stroke edit: re-seed nodes with the colour model fixed; the residual
// graph stays, only e moves by the change of cs - ct (indices unique).
// Duplicate indices in one edit list: the last entry of a node wins.  The
// height plane is scratch between solves (every solve starts with a global
// relabel that rewrites it), so it records the winning entry per node:
// mark -1 on every edited node, then atomicMax of the entry index.
__device__ __forceinline__ long long padded_of(const GridDev& g, long long i) {
  const int x = (int)(i % g.W);
  const long long yz = i / g.W;
  const int y = (int)(yz % g.H), z = (int)(yz / g.H);
  return (long long)x + (long long)g.pitch * (y + (long long)g.Hp * z);
}

__global__ void k_edit_mark(GridDev g, const uint32_t* __restrict__ idx, long long n, int last) {
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n;
       j += (long long)gridDim.x * blockDim.x) {
    int* h = g.h + padded_of(g, idx[j]);
    if (last) atomicMax(h, (int)j);
    else *h = -1;
  }
}

template <int PF>
__global__ void k_edit_seeds(GridDev g, const void* __restrict__ img, uint8_t* __restrict__ seeds,
                             BuildModelDev m, const int* __restrict__ mu, const int* __restrict__ lut_t,
                             const uint32_t* __restrict__ idx, const uint8_t* __restrict__ nseed, long long n,
                             long long* dsink) {
  __shared__ TlinkModel<PF> s_m;
  load_model<PF>(s_m, m, mu);
  __syncthreads();
  long long acc = 0;
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n;
       j += (long long)gridDim.x * blockDim.x) {
    const long long i = idx[j];
    if (g.h[padded_of(g, i)] != (int)j) continue;   // a later entry edits this node
    const int s1 = nseed[j], s0 = seeds[i];
    if (s0 == s1) continue;
    int f[1][3] = {{0, 0, 0}}, cs0[1], ct0[1], cs1[1], ct1[1];
    feat<PF>(img, i, f[0]);
    const int from[1] = {s0}, to[1] = {s1};
    tlinks<PF, 1>(s_m, m.seed_cap, lut_t, f, from, cs0, ct0);
    tlinks<PF, 1>(s_m, m.seed_cap, lut_t, f, to, cs1, ct1);
    int x, y, z;
    dense_xyz(g, i, x, y, z);
    const long long p = (long long)x + (long long)g.pitch * (y + (long long)g.Hp * z);
    atomicAdd(g.e + p, (cs1[0] - ct1[0]) - (cs0[0] - ct0[0]));
    acc += (long long)ct1[0] - ct0[0];
    seeds[i] = (uint8_t)s1;
  }
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
  if ((threadIdx.x & 31) == 0 && acc) atomicAdd((unsigned long long*)dsink, (unsigned long long)acc);
}

int flat_blocks(long long n) {
  long long b = (n + 255) / 256;
  if (b > 148 * 16) b = 148 * 16;
  if (b < 1) b = 1;
  return (int)b;
}

}  // namespace

cudaError_t launch_contrast_sum(const GridDev& g, const void* d_img, int pixfmt,
                                unsigned long long* d_sum, cudaStream_t s) {
  const long long bytes = (long long)g.W * g.H * g.D * (long long)jfc_pix_bytes(pixfmt);
  const int nb = (int)std::max<long long>(1, std::min<long long>((bytes + 16 * 256 - 1) / (16 * 256), 148 * 8));
  const bool d3 = g.dims == 3;
  jfc_note_launch();
  switch (pixfmt) {
    case JFC_PIX_GRAY8: d3 ? k_contrast_sum<JFC_PIX_GRAY8, 3><<<nb, 256, 0, s>>>(g, d_img, d_sum)
                           : k_contrast_sum<JFC_PIX_GRAY8, 2><<<nb, 256, 0, s>>>(g, d_img, d_sum); break;
    case JFC_PIX_RGB8: d3 ? k_contrast_sum<JFC_PIX_RGB8, 3><<<nb, 256, 0, s>>>(g, d_img, d_sum)
                          : k_contrast_sum<JFC_PIX_RGB8, 2><<<nb, 256, 0, s>>>(g, d_img, d_sum); break;
    case JFC_PIX_I16: d3 ? k_contrast_sum<JFC_PIX_I16, 3><<<nb, 256, 0, s>>>(g, d_img, d_sum)
                         : k_contrast_sum<JFC_PIX_I16, 2><<<nb, 256, 0, s>>>(g, d_img, d_sum); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_seed_stats(const GridDev& g, const void* d_img, int pixfmt, const uint8_t* d_seeds,
                              int* d_minmax, unsigned long long* d_count, uint32_t* d_list_f,
                              uint32_t* d_list_b, unsigned int* d_fill, bool fill, cudaStream_t s) {
  if (reinterpret_cast<uintptr_t>(d_seeds) & 15) return cudaErrorMisalignedAddress;   // 16-byte vector loads
  const int nb = flat_blocks(((long long)g.W * g.H * g.D + 15) / 16);
  switch (pixfmt) {
    case JFC_PIX_GRAY8:
      jfc_note_launch();
      k_seed_stats<JFC_PIX_GRAY8><<<nb, 256, 0, s>>>(g, d_img, d_seeds, d_minmax, d_count, d_list_f, d_list_b, d_fill, fill);
      break;
    case JFC_PIX_RGB8:
      jfc_note_launch();
      k_seed_stats<JFC_PIX_RGB8><<<nb, 256, 0, s>>>(g, d_img, d_seeds, d_minmax, d_count, d_list_f, d_list_b, d_fill, fill);
      break;
    case JFC_PIX_I16:
      jfc_note_launch();
      k_seed_stats<JFC_PIX_I16><<<nb, 256, 0, s>>>(g, d_img, d_seeds, d_minmax, d_count, d_list_f, d_list_b, d_fill, fill);
      break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <int PF>
static cudaError_t kmeans_t(const uint32_t* d_list, KmeansDev* d_km, unsigned long long ntotal, int iters,
                            cudaStream_t s) {
  // A cluster of up to 8 blocks while its 8,192 threads have at most 16 seeds
  // each (an iteration of 16 seeds a thread takes about what the grid barrier
  // and the global sums of the other form take, 7 us).  Longer lists take the
  // whole GPU.
  constexpr unsigned long long kClusterSeeds = 8ull * kKmThreads * 16;
  jfc_note_launch();
  if (ntotal <= kClusterSeeds) {
    unsigned blocks = 1;
    while (blocks < 8 && (unsigned long long)blocks * kKmThreads < ntotal) blocks *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kKmThreads);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = blocks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_kmeans<PF, true>, d_list, d_km, iters);
  }
  static int cache[64] = {0};
  const void* fn = (const void*)k_kmeans<PF, false>;
  const int blocks = persistent_blocks_cached(cache, fn, kKmThreads);
  void* params[] = {(void*)&d_list, (void*)&d_km, (void*)&iters};
  return cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(kKmThreads), params, 0, s);
}

cudaError_t launch_kmeans(const uint32_t* d_list, KmeansDev* d_km, int pixfmt, unsigned long long ntotal,
                          int iters, cudaStream_t s) {
  switch (pixfmt) {
    case JFC_PIX_GRAY8: return kmeans_t<JFC_PIX_GRAY8>(d_list, d_km, ntotal, iters, s);
    case JFC_PIX_RGB8: return kmeans_t<JFC_PIX_RGB8>(d_list, d_km, ntotal, iters, s);
    case JFC_PIX_I16: return kmeans_t<JFC_PIX_I16>(d_list, d_km, ntotal, iters, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_expand_runs(const int* d_start, const int* d_val, int m, int n, int* d_out, uint8_t* d_out8,
                               cudaStream_t s) {
  if (n <= 0 || m <= 0) return cudaErrorInvalidValue;
  jfc_note_launch();
  k_expand_runs<<<(n + 255) / 256, 256, 0, s>>>(d_start, d_val, m, n, d_out, d_out8);
  return cudaGetLastError();
}

// Shared memory of k_build's byte tables; the pass uses them while two blocks
// of it fit an SM (one block of 16 warps does not hide the look-ups' latency).
static size_t build_table_bytes(int dims, int nxy, int nz) {
  return (size_t)pad16(JFC_TQ + 1) + pad16(nxy) + (dims == 3 ? pad16(nz) : 0);
}
bool build_tables_fit(int dims, int nxy, int nz) { return build_table_bytes(dims, nxy, nz) <= 108 * 1024; }

template <int PF, int DIMS, bool BYTES>
static cudaError_t build_t(const GridDev& g, const void* d_img, const uint8_t* d_seeds, const BuildModelDev& m,
                           const int* d_mu, const BuildTables& tb, unsigned long long* d_sink, cudaStream_t s) {
  const void* fn = (const void*)k_build<PF, DIMS, BYTES>;
  const size_t dyn = BYTES ? build_table_bytes(DIMS, tb.nxy, tb.nz) : 0;
  if (BYTES) {
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 108 * 1024);
    if (e != cudaSuccess) return e;
  }
  // strips of 16 rows, or of 4 or 1 while those would not give every SM 24 warps
  const int cols = (g.pitch + 127) / 128, warps = kBuildThreads / 32;
  auto strips = [&](int rows) { return (long long)cols * ((g.Hp + rows - 1) / rows) * g.Dp; };   // a warp each
  const int rows = strips(16) >= 148 * 24 ? 16 : strips(4) >= 148 * 24 ? 4 : 1;
  const int grid = (int)std::min<long long>((strips(rows) + warps - 1) / warps, 148 * 2);
  jfc_note_launch();
  k_build<PF, DIMS, BYTES><<<grid, kBuildThreads, dyn, s>>>(g, d_img, d_seeds, m, d_mu, tb, rows, d_sink);
  return cudaGetLastError();
}

cudaError_t launch_build_graph(const GridDev& g, const void* d_img, const uint8_t* d_seeds, const BuildModelDev& m,
                               const int* d_mu, const NlinkTables& nl, const int* d_lut_t, const uint8_t* d_lut_t8,
                               unsigned long long* d_sink, cudaStream_t s) {
  BuildTables tb{nl.xy, nl.z, d_lut_t, nl.xy8, nl.z8, d_lut_t8, nl.nxy, nl.nz};
  const bool d3 = g.dims == 3, bytes = nl.xy8 != nullptr;
#define JFC_BUILD(PF)                                                                                       \
  return d3 ? (bytes ? build_t<PF, 3, true>(g, d_img, d_seeds, m, d_mu, tb, d_sink, s)                      \
                     : build_t<PF, 3, false>(g, d_img, d_seeds, m, d_mu, tb, d_sink, s))                    \
            : (bytes ? build_t<PF, 2, true>(g, d_img, d_seeds, m, d_mu, tb, d_sink, s)                      \
                     : build_t<PF, 2, false>(g, d_img, d_seeds, m, d_mu, tb, d_sink, s))
  switch (m.pixfmt) {
    case JFC_PIX_GRAY8: JFC_BUILD(JFC_PIX_GRAY8);
    case JFC_PIX_RGB8: JFC_BUILD(JFC_PIX_RGB8);
    case JFC_PIX_I16: JFC_BUILD(JFC_PIX_I16);
    default: return cudaErrorInvalidValue;
  }
#undef JFC_BUILD
}

cudaError_t launch_edit_seeds(const GridDev& g, const void* d_img, uint8_t* d_seeds, const BuildModelDev& m,
                              const int* d_mu, const int* d_lut_t, const uint32_t* d_idx,
                              const uint8_t* d_new, size_t n, long long* d_dsink, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const int nb = flat_blocks((long long)n);
  jfc_note_launch(2);
  k_edit_mark<<<nb, 256, 0, s>>>(g, d_idx, (long long)n, 0);
  k_edit_mark<<<nb, 256, 0, s>>>(g, d_idx, (long long)n, 1);
  switch (m.pixfmt) {
    case JFC_PIX_GRAY8:
      jfc_note_launch();
      k_edit_seeds<JFC_PIX_GRAY8><<<nb, 256, 0, s>>>(g, d_img, d_seeds, m, d_mu, d_lut_t, d_idx, d_new, (long long)n, d_dsink);
      break;
    case JFC_PIX_RGB8:
      jfc_note_launch();
      k_edit_seeds<JFC_PIX_RGB8><<<nb, 256, 0, s>>>(g, d_img, d_seeds, m, d_mu, d_lut_t, d_idx, d_new, (long long)n, d_dsink);
      break;
    case JFC_PIX_I16:
      jfc_note_launch();
      k_edit_seeds<JFC_PIX_I16><<<nb, 256, 0, s>>>(g, d_img, d_seeds, m, d_mu, d_lut_t, d_idx, d_new, (long long)n, d_dsink);
      break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}
