// How the DTS passes cut an instance's lines (dts_passes.cu, dts_bounds.cu),
// from its own size and the halo alone: the fixed-point scale of a window sum
// comes from the largest magnitude in its segment, so an image has the same
// bits alone and in a batch.  (Without divisions: a thread has a dozen pixels
// to do.)
#pragma once

#include <cuda_runtime.h>

namespace dtsgb {

constexpr int kXWarps = 4;  // row segments of an X block, each a warp's own

// X: a warp takes a segment of tw pixels of a row and its halo, in rounds of
// 128 columns that it holds in registers: long segments repeat less halo,
// short ones spread an image that is too small for the SMs.
constexpr int kRoundsX = 4, kRoundsWide = 8;  // Wide: halos that need more
struct XGeom {
  int tw, ha, halo;  // segment, left halo, both halos
};
__host__ __device__ inline int x_rounds(int w, int h, int halo) {
  const long long px = (long long)w * h;
  const int need = (halo + 127) / 128 + 1;  // rounds of a segment of 128 pixels
  const int want = px < (1 << 16) ? 2 : px < (1 << 19) ? 3 : kRoundsX;
  return need <= 2 ? want : need == 3 ? kRoundsX : kRoundsWide;
}
__host__ __device__ inline XGeom x_geom(int w, int h, int hx) {
  XGeom g;
  g.ha = (hx + 4) & ~3;
  g.halo = g.ha + ((hx + 3) & ~3);
  g.tw = 128 * x_rounds(w, h, g.halo) - g.halo;
  return g;
}
// Y: tiles of 32 columns x th rows, th + 2hy a multiple of the rows that a warp
// of the launch holds in registers (8, 16 or 32: the tile, and so the result,
// does not depend on which).
__host__ __device__ inline int y_lg(int hy) { return hy <= 56 ? 4 : 5; }
__host__ __device__ inline int y_th(int w, int h, int hy) {
  const long long px = (long long)w * h;
  const int lg = y_lg(hy);
  // up to 16 warps of 16 rows; more where the halo would be most of the tile
  const int full = hy <= 16 ? 8 : hy <= 56 ? 16 : hy <= 127 ? 12 : hy <= 200 ? 16 : 20;
  const int want = px < (1 << 16) ? 32 : 64;  // rows of a tile of a small image
  int warps = (want + 2 * hy + (1 << lg) - 1) >> lg;
  if (px >= (1 << 19) || warps > full) warps = full;
  return (warps << lg) - 2 * hy;
}

// Entry t of a row segment: entry t & 3 of quad t >> 2, one plane of quads per
// entry of a quad, so that the lanes of a warp (a quad each) read and write 32
// banks.  Byte offset t + (t & 3) * (4 QS - 1), QS words a plane (and room for
// 32 entries past the rounds).
template <int NR>
struct XPrefix {
  static constexpr int QS = NR * 32 + 8;
  static __device__ __forceinline__ unsigned* entry(char* S, int t) {
    return reinterpret_cast<unsigned*>(S + t + (t & 3) * (4 * QS - 1));
  }
  static __device__ __forceinline__ unsigned at(const char* S, int t) {
    return *reinterpret_cast<const unsigned*>(S + t + (t & 3) * (4 * QS - 1));
  }
};

// A window's radii from the low byte of a packed word, held to the staged halo:
// whatever the plane holds, no window reads outside its tile.
__device__ __forceinline__ int radius_l(unsigned b, int halo) {
  return min((int)(b & 0xff), halo + 1);
}
__device__ __forceinline__ int radius_u(unsigned b, int halo) {
  return min((int)(b & 0xff), halo);
}
// Its pixels, dl + du from the low two bytes, for the table of 1/n alone.
__device__ __forceinline__ int window_count(unsigned b, int halo) {
  return min((int)((b & 0xff) + ((b >> 8) & 0xff)), 2 * halo + 1);
}

// The passes' grids over a launch's instances (one instance: from its size;
// several: the block tables of launch_pass_blocks for this halo), and the rounds
// and staged rows of the largest.
struct PassGrid {
  dim3 x, y;
  int rounds = 1, rows = 1;
  long long px = 0;
};
struct DtsLaunch;
PassGrid pass_grid(const DtsLaunch& L, int hx, int hy);

}  // namespace dtsgb
