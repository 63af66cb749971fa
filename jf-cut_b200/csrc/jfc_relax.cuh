// jfc_relax.cuh — CTA tile geometry, the arc bits of the 3D global relabel, closures of row words.
#pragma once

#include "jfc_sync.cuh"

namespace jfc {

// One CTA per tile of 32 x TY (x TZ) nodes, one thread per node, one warp per
// tile row.  Heights live in a shared-memory box with a one-cell halo; a row
// of the box is HX_ wide and node x of the tile sits at column x + X0_ (the
// push-relabel visit uses a 40-wide box starting 4 columns left of the tile,
// the shape its tensor-copy staging lands in).
template <int DIMS, int TY_, int TZ_, int HX_ = 34, int X0_ = 1>
struct CtaTile {
  static constexpr int D = DIMS, TY = TY_, TZ = TZ_;
  static constexpr int R = TY * TZ;            // rows = warps
  static constexpr int NT = 32 * R;            // threads = nodes
  static constexpr int K = DIMS == 2 ? 4 : 6;  // arcs per node
  static constexpr int HX = HX_, X0 = X0_, HY = TY + 2, HZ = DIMS == 3 ? TZ + 2 : 1;
  static constexpr int HN = HX * HY * HZ;
  static constexpr int SY = HX, SZ = HX * HY; // box strides
  // arc slots (reference channel order)
  static constexpr int XP = 0, YP = 1;
  static constexpr int ZP = DIMS == 2 ? 0 : 2, ZM = DIMS == 2 ? 0 : 3;
  static constexpr int YM = DIMS == 2 ? 2 : 4, XM = DIMS == 2 ? 3 : 5;
  // halo cells: y faces (2 x TZ x 32), x faces (2 x R), z faces (2 x TY x 32)
  static constexpr int NHY = 2 * TZ * 32, NHX = 2 * R, NHZ = DIMS == 3 ? 2 * TY * 32 : 0;
  static constexpr int NHALO = NHY + NHX + NHZ;
  __device__ static constexpr int hidx(int x, int y, int z) {
    return ((DIMS == 3 ? (z + 1) * HY : 0) + (y + 1)) * HX + (x + X0);
  }
  // halo cell c -> (x, y, z) relative to the tile origin and its face
  // (0 x-, 1 x+, 2 y-, 3 y+, 4 z-, 5 z+)
  __device__ static void halo_cell(int c, int& x, int& y, int& z, int& face) {
    if (c < NHY) {
      const int side = c / (TZ * 32), k = c % (TZ * 32);
      x = k & 31; z = k >> 5; y = side ? TY : -1; face = side ? 3 : 2;
    } else if (c < NHY + NHX) {
      const int k = c - NHY, side = k / R, row = k % R;
      x = side ? 32 : -1; y = row % TY; z = row / TY; face = side ? 1 : 0;
    } else {
      const int k = c - NHY - NHX, side = k / (TY * 32), m = k % (TY * 32);
      x = m & 31; y = m >> 5; z = side ? TZ : -1; face = side ? 5 : 4;
    }
  }
};

// Arc bits used by the relaxation: bit 0 +x, 1 +y, 2 -y, 3 -x, 4 +z, 5 -z.
constexpr unsigned A_XP = 1u, A_YP = 2u, A_YM = 4u, A_XM = 8u, A_ZP = 16u, A_ZM = 32u;

// bit x reached from bit x - 1 (x + 1) when m bit x is set; closure by doubling
__device__ __forceinline__ unsigned close_right(unsigned p, unsigned m) {
  p |= (p << 1) & m; m &= m << 1;
  p |= (p << 2) & m; m &= m << 2;
  p |= (p << 4) & m; m &= m << 4;
  p |= (p << 8) & m; m &= m << 8;
  p |= (p << 16) & m;
  return p;
}
__device__ __forceinline__ unsigned close_left(unsigned p, unsigned m) {
  p |= (p >> 1) & m; m &= m >> 1;
  p |= (p >> 2) & m; m &= m >> 2;
  p |= (p >> 4) & m; m &= m >> 4;
  p |= (p >> 8) & m; m &= m >> 8;
  p |= (p >> 16) & m;
  return p;
}

}  // namespace jfc
