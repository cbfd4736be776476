// Window bounds (a4): the ends of every pixel's window along its row and its
// column, one word per pixel (dl_x | du_x << 8 | dl_y << 16 | du_y << 24).
// Lower bound: the largest i < p with sum_{j=i+1..p} w(j) > sigma, else p-1.
// Upper bound: (the smallest i > p, i < limit, with sum_{j=p+1..i} w(j) >
// sigma) - 1, else p (src/domain_transform_filter.cuh:7-28).  limit is W for X
// and min(W,H) (reference quirk) or H for Y.  A negative ratio stands for an
// all-zero domain transform (no differential computed yet): every window is
// the pixel itself.
//
// The weights are clamped to sigma + 1 (a window holding a larger one
// exceeds sigma either way) and converted to fixed point at 2^F with
// r * (sigma + 1) * 2^F <= 2^30, so a window sum is the exact difference of
// two wrapping 32-bit prefixes of the converted weights (each within 2^-F-1
// of the float weight: decisions differ from float sums only within about
// r * 2^-F of the threshold).
//
// A pass along rows, then one down columns, cut as the iteration's passes are
// (dts_geom.cuh), so that a weight is computed little more than once: 32 x 32
// tiles took it 1.6 times at radius 9 and 5 times at 65.  A pixel's ends are
// found by a binary search over the radius in the prefix, four pixels at a
// time: the steps are the same for every lane, where two pointers that advance
// along a segment made a warp wait for its longest advance at every pixel.
// Bound by issue slots (540 instructions a pixel in tiles with two pointers;
// here 160 and 162 at radius 9, 86% and 81% of the slots busy).
#include <algorithm>
#include <cmath>

#include "../../include/dtsgb.h"
#include "dts_geom.cuh"
#include "dtsgb_internal.cuh"

namespace dtsgb {
namespace {

// The weight between two pixels of a line in fixed point.
struct Weight {
  float ratio, cap, scale;
  int T;  // floor(sigma * 2^F)
  __device__ __forceinline__ unsigned operator()(unsigned a, unsigned b) const {
    return (unsigned)__float2int_rn(
        fminf(edge_weight(*reinterpret_cast<const uchar4*>(&a),
                          *reinterpret_cast<const uchar4*>(&b), ratio),
              cap) *
        scale);
  }
};

// The window ends dl | du << 8 of N pixels of a line.  at(k): pixel k's prefix
// entry, entries STRIDE bytes apart; a distance grows by at least 1 a pixel, so
// sigma ends a window within h = floor(sigma) pixels of its centre, and the
// weights of pixels outside the image (and of pixel 0, which joins no window
// from the left) are zero, so that a search that runs over the border finds
// nothing there.
template <int STRIDE, int N, typename AT>
__device__ __forceinline__ void window_ends(int h, int T, AT&& at, const int (&p)[N], int lim,
                                            unsigned (&ends)[N]) {
  const char *c[N], *lo[N], *hi[N];
  unsigned s[N];  // (the prefixes wrap: only their differences are signed)
#pragma unroll
  for (int k = 0; k < N; ++k) {
    c[k] = lo[k] = hi[k] = at(k);
    s[k] = *reinterpret_cast<const unsigned*>(c[k]);
  }
  // the farthest entries within T, h >= 0 pixels away at most
  for (int n = h; n > 0; n >>= 1) {
    const int step = ((n + 1) >> 1) * STRIDE;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const char *l = lo[k] - step, *u = hi[k] + step;
      if ((int)(s[k] - *reinterpret_cast<const unsigned*>(l)) <= T) lo[k] = l;
      if ((int)(*reinterpret_cast<const unsigned*>(u) - s[k]) <= T) hi[k] = u;
    }
  }
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const int dl = (int)(c[k] - lo[k]) / STRIDE, du = (int)(hi[k] - c[k]) / STRIDE;
    // no pixel of the line exceeds sigma on that side: the window stops short
    ends[k] = (unsigned)(dl >= p[k] ? 1 : dl + 1) | (du >= lim - 1 - p[k] ? 0u : (unsigned)du << 8);
  }
}

// A warp per row segment: its weights from registers (four adjacent pixels a
// lane and round), a shuffle scan per round, then 4 x 32 pixels at a time.
template <int NR>
__global__ void __launch_bounds__(32 * kXWarps)
    k_bounds_x(const Inst* __restrict__ insts, const uchar4* __restrict__ guide,
               uint32_t* __restrict__ bounds, Weight wt, int hx,
               const Tile* __restrict__ blocks) {
  extern __shared__ __align__(16) unsigned smx[];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned* S = smx + warp * (128 * NR);
  const Tile t = blocks ? blocks[blockIdx.x] : Tile{0, (int)blockIdx.y, (int)blockIdx.x, 0};
  const Inst in = insts[t.inst];
  const int W = in.w;
  const XGeom g = x_geom(W, in.h, hx);
  const int row = t.y0 * kXWarps + warp, x0 = t.x0 * g.tw;
  if (row >= in.h) return;
  const int xe = min(x0 + g.tw, W);
  const long long base = in.off + (long long)row * in.pitch;
  uint32_t* out = bounds + base;
  if (wt.ratio < 0.f) {
    for (int x = x0 + lane; x < xe; x += 32) out[x] = 1u;
    return;
  }
  const int rounds = (xe - x0 + g.halo + 127) >> 7;
  const int xl = x0 - g.ha + 4 * lane;  // the lane's first pixel of round 0
  uint4 c[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const int x = xl + 128 * r;
    c[r] = make_uint4(0u, 0u, 0u, 0u);
    if (x >= 0 && x < W && r < rounds)
      c[r] = __ldg(reinterpret_cast<const uint4*>(guide + (base + x)));
  }
  unsigned carry = 0u, left = 0u;  // the prefix and the pixel before the round
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    if (r < rounds) {
      const int x = xl + 128 * r;
      unsigned prev = __shfl_up_sync(0xffffffffu, c[r].w, 1);
      if (lane == 0) prev = left;
      left = __shfl_sync(0xffffffffu, c[r].w, 31);
      // (the first entry of the segment begins no distance: its weight is free)
      uint4 a;
      a.x = x > 0 && x < W ? wt(c[r].x, prev) : 0u;
      a.y = a.x + (x >= 0 && x + 1 < W ? wt(c[r].y, c[r].x) : 0u);
      a.z = a.y + (x >= 0 && x + 2 < W ? wt(c[r].z, c[r].y) : 0u);
      a.w = a.z + (x >= 0 && x + 3 < W ? wt(c[r].w, c[r].z) : 0u);
      unsigned incl = a.w;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
      }
      const unsigned off = carry + incl - a.w;
      reinterpret_cast<uint4*>(S)[lane + 32 * r] =
          make_uint4(off + a.x, off + a.y, off + a.z, off + a.w);
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
  __syncwarp();
  for (int x = x0 + lane; x < xe; x += 128) {
    int p[4];
    unsigned e[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) p[k] = min(x + 32 * k, xe - 1);
    window_ends<4, 4>(
        hx, wt.T, [&](int k) { return reinterpret_cast<const char*>(S + (p[k] - x0 + g.ha)); },
        p, W, e);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (x + 32 * k < xe) out[x + 32 * k] = e[k];
  }
}

// A block per 32 columns x th rows, lanes on columns; a warp computes the
// weights of RM staged rows, the prefixes are joined through shared memory and
// a warp searches for the tile rows that it holds.  It adds its half to the
// words that the X pass wrote.
template <int RM>
__global__ void __launch_bounds__(RM == 32 ? 768 : 512, RM == 32 ? 1 : 2)
    k_bounds_y(const Inst* __restrict__ insts, const uchar4* __restrict__ guide,
               uint32_t* __restrict__ bounds, Weight wt, int hy, int ref_y_limit,
               const Tile* __restrict__ blocks) {
  extern __shared__ unsigned smy[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const Tile t = blocks ? blocks[blockIdx.x] : Tile{0, (int)blockIdx.x, (int)blockIdx.y, 0};
  const Inst in = insts[t.inst];
  const int W = in.w, H = in.h, P = in.pitch;
  const int th = y_th(W, H, hy), warps = (th + 2 * hy) / RM;
  const int x = t.x0 * 32 + lane, y0 = t.y0 * th;
  unsigned* tot = smy;                 // warps x 32
  unsigned* S = tot + warps * 32;      // staged rows x 32
  if (warp >= warps) return;           // (whole warps; see the barriers)
  const int live = 32 * warps;         // threads at the barriers
  const bool inx = x < W;
  const int s0 = warp * RM;            // the warp's first staged row
  const int ys = y0 - hy + s0;         // its image row
  const int jm = min(th, H - y0);      // tile rows
  const long long first = in.off + (long long)ys * P + x;
  const int k0 = max(hy - s0, 0), k1 = min(jm + hy - s0, RM);  // tile rows it holds
  uint16_t* out = reinterpret_cast<uint16_t*>(bounds + first) + 1;
  if (wt.ratio < 0.f) {
    pdl_wait_then_release();
    for (int k = k0; k < k1; ++k)
      if (inx) out[2 * (long long)k * P] = 1u;
    return;
  }
  {
    const unsigned* gc = reinterpret_cast<const unsigned*>(guide) + first;
    unsigned v[RM + 1];
#pragma unroll
    for (int k = 0; k <= RM; ++k)
      v[k] = inx && (unsigned)(ys + k - 1) < (unsigned)H ? __ldg(gc + (long long)(k - 1) * P) : 0u;
    unsigned a[RM], acc = 0u;
#pragma unroll
    for (int k = 0; k < RM; ++k) {
      if (ys + k > 0 && ys + k < H) acc += wt(v[k + 1], v[k]);
      a[k] = acc;
    }
    tot[warp * 32 + lane] = acc;
    asm volatile("bar.sync 1, %0;" ::"r"(live) : "memory");
    unsigned off = 0u;
    for (int w = 0; w < warp; ++w) off += tot[w * 32 + lane];
#pragma unroll
    for (int k = 0; k < RM; ++k) S[(s0 + k) * 32 + lane] = off + a[k];
  }
  asm volatile("bar.sync 1, %0;" ::"r"(live) : "memory");
  pdl_wait_then_release();  // the X pass wrote its half
  if (!inx) return;
  const int lim = ref_y_limit ? min(W, H) : H;
  for (int k = k0; k < k1; k += 4) {
    int p[4];
    unsigned e[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) p[j] = ys + min(k + j, k1 - 1);
    window_ends<128, 4>(
        hy, wt.T,
        [&](int j) {
          return reinterpret_cast<const char*>(S + (p[j] - y0 + hy) * 32 + lane);
        },
        p, lim, e);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (k + j < k1) out[2 * (long long)(k + j) * P] = (uint16_t)e[j];
  }
}

template <int NR>
int launch_x(const DtsLaunch& L, const PassGrid& G, const uchar4* guide, uint32_t* bounds,
             const Weight& wt, int hx, cudaStream_t s) {
  k_bounds_x<NR><<<G.x, 32 * kXWarps, sizeof(unsigned) * kXWarps * 128 * NR, s>>>(
      L.d_inst, guide, bounds, wt, hx, L.n_inst > 1 ? L.d_xblocks : nullptr);
  DTSGB_CUDA(cudaGetLastError());
  return DTSGB_OK;
}

template <int RM>
int launch_y(const DtsLaunch& L, const PassGrid& G, const uchar4* guide, uint32_t* bounds,
             const Weight& wt, int hy, int ref_y_limit, cudaStream_t s) {
  auto kern = k_bounds_y<RM>;
  const int warps = G.rows / RM;
  const size_t smem = sizeof(unsigned) * 32 * (size_t)(warps + G.rows);
  DTSGB_CUDA(allow_smem(kern, smem));
  DTSGB_CUDA(launch_dependent(kern, G.y, dim3(32 * warps), smem, s, L.d_inst, guide, bounds, wt,
                              hy, ref_y_limit, L.n_inst > 1 ? L.d_yblocks : (const Tile*)nullptr));
  return DTSGB_OK;
}

}  // namespace

int launch_bounds(const DtsLaunch& L, const uchar4* guide, uint32_t* bounds,
                  float ratio_x, float ratio_y, float sigma_x, float sigma_y,
                  int ref_y_limit, cudaStream_t s) {
  const int rx = (int)floorf(sigma_x) + 1, ry = (int)floorf(sigma_y) + 1;
  if (rx > 255 || ry > 255)
    return fail(DTSGB_ERR_UNSUPPORTED, "sigma >= 255 is not supported");
  if (L.one_by_one()) {
    for (int i = 0; i < L.n_inst; ++i)
      if (int e = launch_bounds(L.one(i), guide, bounds, ratio_x, ratio_y, sigma_x, sigma_y,
                                ref_y_limit, s))
        return e;
    return DTSGB_OK;
  }
  // fixed point per axis: r * (sigma + 1) * 2^F <= 2^30; threshold floor(sigma 2^F)
  auto fx = [](int r, float sigma, float ratio) {
    Weight w;
    w.ratio = ratio;
    w.cap = sigma + 1.f;
    const int F = 30 - (int)std::ceil(std::log2((double)r * (double)w.cap));
    w.scale = std::ldexp(1.f, F);
    w.T = (int)std::floor((double)sigma * std::ldexp(1.0, F));
    return w;
  };
  const Weight wx = fx(rx, sigma_x, ratio_x), wy = fx(ry, sigma_y, ratio_y);
  const int hx = rx - 1, hy = ry - 1;
  const PassGrid G = pass_grid(L, hx, hy);
  ProfScope ps(s, DTSGB_K_BOUNDS);
  int st;
  if (G.rounds <= 2) st = launch_x<2>(L, G, guide, bounds, wx, hx, s);
  else if (G.rounds <= 3) st = launch_x<3>(L, G, guide, bounds, wx, hx, s);
  else if (G.rounds <= kRoundsX) st = launch_x<kRoundsX>(L, G, guide, bounds, wx, hx, s);
  else st = launch_x<kRoundsWide>(L, G, guide, bounds, wx, hx, s);
  if (st) return st;
  // the rows a warp holds: as the iteration's Y pass
  if (G.rows <= 128 && G.px < (4 << 20))
    return launch_y<8>(L, G, guide, bounds, wy, hy, ref_y_limit, s);
  return G.rows <= 256 ? launch_y<16>(L, G, guide, bounds, wy, hy, ref_y_limit, s)
                       : launch_y<32>(L, G, guide, bounds, wy, hy, ref_y_limit, s);
}

}  // namespace dtsgb
