// The DTS iteration (a6/a7) as two passes over memory: the X half-step along
// rows, the Y half-step down columns.
//   X: v' = v - s*(lambda*(v - B_x) + 0.5*g),
//      g = 2*(c/n)*(v - t) (L2) or (c/n)*(v-t)/sqrt((v-t)^2 + 1e-6)
//   Y: v' = v - s*lambda*(v - B_y)
// (src/domain_transform_solver.cuh:12-116).  With overwrite in (0,1), the
// target replaces v where c > overwrite before each half-step
// (src/domain_transform_solver.cu:126-130, 160-164): the X pass does so to
// its results, the Y pass of an iteration that feeds another one to its
// outputs, and the first iterate is the target everywhere.
//
// Window sums are differences of fixed-point prefix sums (fixed_point.cuh)
// along a segment of the line that holds the windows of its pixels.
//
// Passes of their own beat one kernel that keeps the X results of a tile in
// shared memory, the form this replaces (16 or 20 B/px of traffic against 28 or
// 32 here): that one has to run X over the vertical halo of each tile too and
// to stage both halos, (2hx + TW) x (2hy + TH), between five block barriers.
// Measured per iteration: 1376x1088 with sigma_z 71: 131 -> 26 us, with 8: 23 ->
// 15.5; 3264x2448 with 30 and overwrite: 147 -> 86; 64 ragged BF16 images (47
// Mpx) with 8: 366 -> 316; 160x120: 6.7 -> 5.8.
//
// Bound by issue slots and latency, half and half (X: 73 instructions a pixel,
// 58% of the slots busy, 45 us; Y: 66, 60%, 39 us at 12.6 Mpx): loads come
// first in a warp and the arithmetic after, and the other warps of an SM fill
// the gap only in part.
#include <algorithm>
#include <cmath>

#include "../../include/dtsgb.h"
#include "dts_geom.cuh"
#include "dtsgb_internal.cuh"
#include "fixed_point.cuh"
#include "raw4.cuh"

namespace dtsgb {
namespace {

constexpr int kNaNBits = 0x7fc00000;

// X half-step update of one pixel (src/domain_transform_solver.cuh:37-86);
// rn = 1/n correctly rounded.
template <int MODE, bool STEREO>
__device__ __forceinline__ float x_update(float v, float B, float tv, float cv, float rn,
                                          float lambda, float step, float extra) {
  const float cn = cv * rn;
  const float d = v - tv;
  // L2: 0.5 * (2 (c/n) d) is (c/n) d exactly (scaling by 2 is exact)
  if (MODE == 0 && !STEREO) return __fmaf_rn(step, -__fmaf_rn(lambda, v - B, cn * d), v);
  float g;
  if (MODE == 0) {
    g = 2.f * cn * d;
  } else {
    g = __fdiv_rn(cn * d, __fsqrt_rn(__fmaf_rn(d, d, 1e-6f)));
  }
  if (STEREO) g += extra;
  return __fmaf_rn(step, -__fmaf_rn(lambda, v - B, 0.5f * g), v);
}

// PhotometricL2LossTerm::operator() (src/domain_transform_loss_term.cuh:
// 20-39) at pixel x of the row at element `row`, for disparity d:
//   lambda_p * 2 * SAD4(left(x), right(xi)) / 255
//     * ((dH_right(xi)^2 - 1) * alpha),   xi = (int)(offset + x - d),
// zero when offset + x - d falls outside [0, W).  dH_right is the right
// image's dHdx, evaluated here from the right guide.
__device__ __forceinline__ float photometric(const StereoArgs& sa, long long row, int x, int W,
                                             float d) {
  const float xr = (sa.offset + (float)x) - d;
  if (!(xr >= 0.f && xr < (float)W)) return 0.f;
  const int xi = (int)xr;
  const uchar4 a = sa.left[row + x], b = sa.right[row + xi];
  const float sad = ((float)abs((int)a.x - (int)b.x) + (float)abs((int)a.y - (int)b.y) +
                     (float)abs((int)a.z - (int)b.z) + (float)abs((int)a.w - (int)b.w)) *
                    (float)0.00392156863;
  float gr = 0.f;
  if (sa.ratio >= 0.f)
    gr = edge_weight(b, xi > 0 ? sa.right[row + xi - 1] : make_uchar4(0, 0, 0, 0), sa.ratio);
  return sa.lam_p * 2.f * sad * (__fmaf_rn(gr, gr, -1.f) * sa.alpha);
}

__device__ __forceinline__ bool finite_bits(float v) { return mag_bits(v) < kNonFiniteBits; }

// ---------------------------------------------------------------------------
// X half-step.  A warp takes a segment of one row: its lanes load the
// segment and its halo as float4 (four adjacent pixels, 128 a round, kept in
// registers), the largest magnitude sets the scale, a shuffle scan per round
// leaves the prefix in the warp's shared memory, and each lane updates the
// pixels it already holds.  AHEAD: the next round's bounds, target and
// confidence are in flight meanwhile (64 registers); without, 48, and ten
// blocks an SM take turns, which is better where there are that many (see
// launch_iter).  Warps are independent.
//
// The window ends come from dts_bounds.cu for the same sigma (dl <= hx + 1, du <=
// hx).  The caller's graphs may leave another sigma's in the plane: radius_l and
// radius_u keep a prefix index within the staged columns then too.
//
// A non-finite value in the segment has no fixed-point form: the warp then
// adds its windows in float, pixel by pixel, and every result that is not
// finite is NaN (never finite garbage).
// ---------------------------------------------------------------------------
template <typename TS, int MODE, bool STEREO, bool OVER, int NR, bool AHEAD>
__global__ void __launch_bounds__(32 * kXWarps, AHEAD ? 1 : 10)
    k_dts_x(const Inst* __restrict__ insts, const float* __restrict__ vin,
            float* __restrict__ vout, const TS* __restrict__ tgt, const TS* __restrict__ cnf,
            const uint32_t* __restrict__ bnd, float lambda, float step, float overwrite, int hx,
            StereoArgs sa, const Tile* __restrict__ blocks) {
  using PX = XPrefix<NR>;
  extern __shared__ unsigned smx[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned* S = smx + warp * (4 * PX::QS);
  const char* Sb = reinterpret_cast<const char*>(S);
  float* rtab = reinterpret_cast<float*>(smx + kXWarps * 4 * PX::QS);  // 1/n
  // (the tables are written before any pass)
  const Tile t = blocks ? blocks[blockIdx.x] : Tile{0, (int)blockIdx.y, (int)blockIdx.x, 0};
  const Inst in = insts[t.inst];
  const int W = in.w;
  const XGeom g = x_geom(W, in.h, hx);
  const int row = t.y0 * kXWarps + warp, x0 = t.x0 * g.tw;
  const int nrt = 2 * hx + 2;
  for (int i = tid; i < nrt; i += 32 * kXWarps) rtab[i] = i ? __frcp_rn((float)i) : 0.f;
  __syncthreads();
  pdl_wait_then_release();  // launched as a dependent of the pass before
  if (row >= in.h) return;
  const int xe = min(x0 + g.tw, W);
  const int rounds = (xe - x0 + g.halo + 127) >> 7;
  const int xl = x0 - g.ha + 4 * lane;  // the lane's first pixel of round 0
  const long long base = in.off + (long long)row * in.pitch;
  const float* vl = vin + (base + xl);
  const uint32_t* bl = bnd + (base + xl);
  const TS *tl = tgt + (base + xl), *cl = cnf + (base + xl);
  struct Quad {
    uint4 b;
    Raw4<TS> tv, cv;
  };
  // this lane's pixels of round r: in the segment
  auto mine = [&](int r) { return xl + 128 * r >= x0 && xl + 128 * r < xe; };
  auto fetch = [&](int r, Quad& Q) {
    if (mine(r)) {
      Q.b = __ldg(reinterpret_cast<const uint4*>(bl + 128 * r));
      Q.tv.load(tl + 128 * r);
      Q.cv.load(cl + 128 * r);
      const int x = xl + 128 * r;
      if (x + 4 > W) {  // columns past the width: the pitch's padding
        if (x + 1 >= W) Q.b.y = 0u;
        if (x + 2 >= W) Q.b.z = 0u;
        Q.b.w = 0u;
      }
    }
  };
  constexpr int NQ = AHEAD ? 2 : 1;
  Quad Q[NQ];
  float4 v[NR];
  if (x0 - g.ha >= 0 && x0 - g.ha + 128 * rounds <= W) {  // the whole warp inside
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      v[r] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < rounds) v[r] = __ldg(reinterpret_cast<const float4*>(vl + 128 * r));
    }
  } else {
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const int x = xl + 128 * r;
      v[r] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (x >= 0 && x < W && r < rounds) {
        v[r] = __ldg(reinterpret_cast<const float4*>(vl + 128 * r));
        if (x + 1 >= W) v[r].y = 0.f;
        if (x + 2 >= W) v[r].z = 0.f;
        if (x + 3 >= W) v[r].w = 0.f;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NQ; ++i) {
    Q[i].b = make_uint4(0u, 0u, 0u, 0u);
    Q[i].tv.zero();
    Q[i].cv.zero();
  }
  if (AHEAD) fetch(0, Q[0]);
  unsigned mb = 0u;
#pragma unroll
  for (int r = 0; r < NR; ++r)
    mb = max(mb, max(max(mag_bits(v[r].x), mag_bits(v[r].y)),
                     max(mag_bits(v[r].z), mag_bits(v[r].w))));
  mb = __reduce_max_sync(0xffffffffu, mb);
  auto store = [&](int r, const float (&o)[4]) {
    const int x = xl + 128 * r;
    float* dst = vout + (base + x);
    if (x + 4 <= W) {
      *reinterpret_cast<float4*>(dst) = make_float4(o[0], o[1], o[2], o[3]);
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (x + k < W) dst[k] = o[k];
    }
  };
  if (mb >= kNonFiniteBits) {  // the whole warp
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      S[0 * PX::QS + lane + 32 * r] = __float_as_uint(v[r].x);
      S[1 * PX::QS + lane + 32 * r] = __float_as_uint(v[r].y);
      S[2 * PX::QS + lane + 32 * r] = __float_as_uint(v[r].z);
      S[3 * PX::QS + lane + 32 * r] = __float_as_uint(v[r].w);
    }
    __syncwarp();
    for (int x = x0 + lane; x < xe; x += 32) {
      const uint32_t b = __ldg(bnd + base + x);
      const int dl = radius_l(b, hx), du = radius_u(b >> 8, hx), t = x - x0 + g.ha;
      float B = 0.f;
      for (int j = t - dl + 1; j <= t + du; ++j) B += __uint_as_float(PX::at(Sb, j));
      const float rn = rtab[dl + du], vv = __uint_as_float(PX::at(Sb, t));
      const float tv = load_f(tgt + base + x), cv = load_f(cnf + base + x);
      float extra = 0.f;
      if (STEREO) extra = photometric(sa, base, x, W, vv);
      float o = x_update<MODE, STEREO>(vv, B * rn, tv, cv, rn, lambda, step, extra);
      if (OVER && cv > overwrite) o = tv;
      vout[base + x] = finite_bits(o) ? o : __int_as_float(kNaNBits);
    }
    return;
  }
  const int F = fx_shift(__uint_as_float(mb), ceil_log2(2 * hx + 1));
  const float sF = pow2f(F), isF = pow2f(-F);
  unsigned carry = 0u;
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    if (r < rounds) {
      const unsigned a0 = fx_from(v[r].x, sF), a1 = a0 + fx_from(v[r].y, sF);
      const unsigned a2 = a1 + fx_from(v[r].z, sF), a3 = a2 + fx_from(v[r].w, sF);
      const unsigned incl = warp_incl_scan(a3, lane);
      const unsigned off = carry + incl - a3;
      S[0 * PX::QS + lane + 32 * r] = off + a0;
      S[1 * PX::QS + lane + 32 * r] = off + a1;
      S[2 * PX::QS + lane + 32 * r] = off + a2;
      S[3 * PX::QS + lane + 32 * r] = off + a3;
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    if (r < rounds) {
      if (!AHEAD) fetch(r, Q[0]);
      if (AHEAD && r + 1 < NR) fetch(r + 1, Q[(r + 1) % NQ]);
      const Quad& q = Q[r % NQ];
      const int t0 = 4 * lane + 128 * r;
      if (mine(r)) {
        float o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t b = u4_get(q.b, k);
          const int dl = radius_l(b, hx), du = radius_u(b >> 8, hx);
          const float rn = rtab[dl + du];
          const float vv = f4_get(v[r], k), tv = q.tv[k], cv = q.cv[k];
          const float B =
              fx_window(PX::at(Sb, t0 + k + du), PX::at(Sb, t0 + k - dl), rn * isF);
          float extra = 0.f;
          if (STEREO) extra = photometric(sa, base, min(xl + 128 * r + k, W - 1), W, vv);
          o[k] = x_update<MODE, STEREO>(vv, B, tv, cv, rn, lambda, step, extra);
          if (OVER && cv > overwrite) o[k] = tv;
        }
        store(r, o);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Y half-step.  A block takes 32 columns x th rows (lanes on columns, so that
// every access of a warp is 128 contiguous bytes); each warp loads RM rows of
// the tile and its halo, and the bounds of those inside the tile, into
// registers, the warps' prefixes are joined through shared memory, and each
// warp updates the tile rows it holds.  hold: outputs keep the X result (the
// target) where c > overwrite.
// ---------------------------------------------------------------------------
template <typename TS, bool OVER, int RM>
__global__ void __launch_bounds__(RM == 32 ? 768 : 512, RM == 8 ? 3 : RM == 16 ? 2 : 1)
    k_dts_y(const Inst* __restrict__ insts, const float* __restrict__ u,
            float* __restrict__ vout, const TS* __restrict__ cnf,
            const uint32_t* __restrict__ bnd, float slam, float overwrite, int hold, int hy,
            const Tile* __restrict__ blocks) {
  extern __shared__ unsigned smy[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = blockDim.x;
  const Tile t = blocks ? blocks[blockIdx.x] : Tile{0, (int)blockIdx.x, (int)blockIdx.y, 0};
  const Inst in = insts[t.inst];
  const int W = in.w, H = in.h, P = in.pitch;
  const int th = y_th(W, H, hy), warps = (th + 2 * hy) / RM;
  const int cx = t.x0, y0 = t.y0 * th;
  const int nrt = 2 * hy + 2;
  unsigned* smax = smy;
  float* rtab = reinterpret_cast<float*>(smy + 1);      // 1/n
  unsigned* tot = smy + 1 + nrt;                        // warps x 32
  unsigned* S = tot + warps * 32;                     // (rows + 1) x 32: prefix, row 0 = 0
  for (int i = tid; i < nrt; i += nt) rtab[i] = i ? __frcp_rn((float)i) : 0.f;
  if (tid == 0) *smax = 0u;
  __syncthreads();
  pdl_wait_then_release();  // launched as a dependent of the X pass
  const int x = cx * 32 + lane;
  if (warp >= warps) return;  // (whole warps; see the barriers)
  const bool inx = x < W;
  const int s0 = warp * RM;            // the warp's first staged row
  const int ys = y0 - hy + s0;         // its image row
  const int jm = min(th, H - y0);    // tile rows
  const long long first = in.off + (long long)ys * P + x;
  const float* uc = u + first;
  const uint32_t* bc = bnd + first;
  constexpr bool kEarly = RM < 32;  // bounds in flight with the values
  float v[RM];
  uint32_t b[kEarly ? RM : 1];
  if (cx * 32 + 32 <= W && ys >= 0 && ys + RM <= H) {  // the whole warp inside
#pragma unroll
    for (int k = 0; k < RM; ++k) v[k] = __ldg(uc + (long long)k * P);
  } else {
#pragma unroll
    for (int k = 0; k < RM; ++k)
      v[k] = inx && (unsigned)(ys + k) < (unsigned)H ? __ldg(uc + (long long)k * P) : 0.f;
  }
  // the warp's rows that lie in the tile: [k0, k1)
  const int k0 = max(hy - s0, 0), k1 = min(jm + hy - s0, RM);
  if (kEarly) {
    if (cx * 32 + 32 <= W && k0 == 0 && k1 == RM) {
#pragma unroll
      for (int k = 0; k < (kEarly ? RM : 0); ++k) b[k] = __ldg(bc + (long long)k * P);
    } else {
#pragma unroll
      for (int k = 0; k < (kEarly ? RM : 0); ++k)
        b[k] = inx && k >= k0 && k < k1 ? __ldg(bc + (long long)k * P) : 0u;
    }
  }
  if (OVER && hold) {  // the pixels that keep their X result: the free low bits
    float c[kEarly ? RM : 1];
#pragma unroll
    for (int k = 0; k < (kEarly ? RM : 0); ++k)
      c[k] = b[k] ? load_f(cnf + (first + (long long)k * P)) : 0.f;
#pragma unroll
    for (int k = 0; k < (kEarly ? RM : 0); ++k)
      b[k] = (b[k] & 0xffff0000u) | (c[k] > overwrite ? 1u : 0u);
  }
  unsigned mb = 0u;
#pragma unroll
  for (int k = 0; k < RM; ++k) mb = max(mb, mag_bits(v[k]));
  mb = __reduce_max_sync(0xffffffffu, mb);
  if (lane == 0) atomicMax(smax, mb);
  if (warp == 0) S[lane] = 0u;
  const int live = 32 * warps;  // threads at the barriers
  asm volatile("bar.sync 1, %0;" ::"r"(live) : "memory");
  const bool bad = *smax >= kNonFiniteBits;
  unsigned* Sw = S + (s0 + 1) * 32 + lane;
  float* oc = vout + first;
  if (bad) {
#pragma unroll
    for (int k = 0; k < RM; ++k) Sw[k * 32] = __float_as_uint(v[k]);
    asm volatile("bar.sync 1, %0;" ::"r"(live) : "memory");
    for (int k = 0; k < RM; ++k) {
      const int j = s0 + k - hy;
      if (!inx || (unsigned)j >= (unsigned)jm) continue;
      const long long p = first + (long long)k * P;
      const uint32_t bb = __ldg(bnd + p) >> 16;
      const int dl = radius_l(bb, hy), du = radius_u(bb >> 8, hy);
      float B = 0.f;
      for (int q = k - dl + 1; q <= k + du; ++q) B += __uint_as_float(Sw[q * 32]);
      const float vv = __uint_as_float(Sw[k * 32]);
      float o = __fmaf_rn(-slam, vv - B * rtab[dl + du], vv);
      if (!finite_bits(o)) o = __int_as_float(kNaNBits);
      if (OVER && hold && load_f(cnf + p) > overwrite) o = vv;
      vout[p] = o;
    }
    return;
  }
  const int F = fx_shift(__uint_as_float(*smax), ceil_log2(2 * hy + 1));
  const float sF = pow2f(F), isF = pow2f(-F);
  {
    unsigned a[RM];
    a[0] = fx_from(v[0], sF);
#pragma unroll
    for (int k = 1; k < RM; ++k) a[k] = a[k - 1] + fx_from(v[k], sF);
    tot[warp * 32 + lane] = a[RM - 1];
    asm volatile("bar.sync 1, %0;" ::"r"(live) : "memory");
    unsigned off = 0u;
    for (int w = 0; w < warp; ++w) off += tot[w * 32 + lane];
#pragma unroll
    for (int k = 0; k < RM; ++k) Sw[k * 32] = off + a[k];
  }
  asm volatile("bar.sync 1, %0;" ::"r"(live) : "memory");
  if (!inx) return;
  const char* Sc = reinterpret_cast<const char*>(Sw);
  const char* rt = reinterpret_cast<const char*>(rtab);
#pragma unroll
  for (int k = 0; k < RM; ++k) {
    if (k >= k0 && k < k1) {
      const uint32_t bk = kEarly ? b[kEarly ? k : 0] : __ldg(bc + (long long)k * P);
      const int dl = radius_l(bk >> 16, hy), du = radius_u(bk >> 24, hy);
      const unsigned hi = *reinterpret_cast<const unsigned*>(Sc + du * 128 + k * 128);
      const unsigned lo = *reinterpret_cast<const unsigned*>(Sc - dl * 128 + k * 128);
      const float rn = *reinterpret_cast<const float*>(rt + (dl + du) * 4);
      const float B = fx_window(hi, lo, rn * isF);
      float o = __fmaf_rn(-slam, v[k] - B, v[k]);
      if (OVER && hold &&
          (kEarly ? (bk & 1u) != 0u : load_f(cnf + (first + (long long)k * P)) > overwrite))
        o = v[k];
      oc[(long long)k * P] = o;
    }
  }
}

// The block tables of several instances: instance blockIdx.y's blocks in rows,
// from the starts that the host has added up.
constexpr int kBlockStarts = 128;
struct BlockStarts {
  int x[kBlockStarts + 1], y[kBlockStarts + 1];
};
__global__ void __launch_bounds__(256)
    k_pass_blocks(const Inst* __restrict__ insts, int first,
                  const __grid_constant__ BlockStarts S, int halo, Tile* __restrict__ x,
                  Tile* __restrict__ y) {
  const int i = blockIdx.y, e = blockIdx.x * 256 + threadIdx.x;
  const Inst in = insts[first + i];
  const int tw = x_geom(in.w, in.h, halo).tw;
  const int xc = (in.w + tw - 1) / tw, yc = (in.w + 31) / 32;
  if (e < S.x[i + 1] - S.x[i]) x[S.x[i] + e] = Tile{first + i, e % xc, e / xc, 0};
  if (e < S.y[i + 1] - S.y[i]) y[S.y[i] + e] = Tile{first + i, e % yc, e / yc, 0};
}

template <typename TS, int MODE, bool STEREO, bool OVER, int NR, bool AHEAD = true>
int launch_x(const DtsLaunch& L, const float* vin, float* vout, const void* target,
             const void* conf, const uint32_t* bounds, float lambda, float step,
             float overwrite, int hx, dim3 grid, const StereoArgs& sa, cudaStream_t s) {
  auto kern = k_dts_x<TS, MODE, STEREO, OVER, NR, AHEAD>;
  const size_t smem = sizeof(unsigned) * (kXWarps * 4 * XPrefix<NR>::QS + 2 * hx + 2);
  ProfScope ps(s, DTSGB_K_DTS_ITER);
  DTSGB_CUDA(launch_dependent(kern, grid, dim3(32 * kXWarps), smem, s, L.d_inst, vin, vout,
                              (const TS*)target, (const TS*)conf, bounds, lambda, step,
                              overwrite, hx, sa,
                              L.n_inst > 1 ? L.d_xblocks : (const Tile*)nullptr));
  return DTSGB_OK;
}

template <typename TS, bool OVER, int RM>
int launch_y(const DtsLaunch& L, const float* u, float* vout, const void* conf,
             const uint32_t* bounds, float slam, float overwrite, int feeds, int hy,
             dim3 grid, int rows, cudaStream_t s) {
  auto kern = k_dts_y<TS, OVER, RM>;
  const int warps = rows / RM;
  const size_t smem = sizeof(unsigned) *
                      ((size_t)(2 * hy + 3) + warps * 32 + ((size_t)rows + 1) * 32);
  DTSGB_CUDA(allow_smem(kern, smem));
  ProfScope ps(s, DTSGB_K_DTS_ITER);
  DTSGB_CUDA(launch_dependent(kern, grid, dim3(32 * warps), smem, s, L.d_inst, u, vout,
                              (const TS*)conf, bounds, slam, overwrite, feeds, hy,
                              L.n_inst > 1 ? L.d_yblocks : (const Tile*)nullptr));
  return DTSGB_OK;
}

template <typename TS, int MODE, bool STEREO, bool OVER>
int launch_iter(const DtsLaunch& L, const float* vin, float* tmp, float* vout, const void* target,
                const void* conf, const uint32_t* bounds, float lambda, float step,
                float overwrite, int feeds, int halo, const StereoArgs& sa, cudaStream_t s) {
  const PassGrid G = pass_grid(L, halo, halo);
  const dim3 gx = G.x, gy = G.y;
  const int rounds = G.rounds, rows = G.rows;
  const long long px = G.px;
  int st;
  // enough blocks to fill the SMs without the loads ahead: 3264x2448 950 -> 898
  // us a solve, 16 x 1024x768 2427 -> 2386 a training step; 1376x1088, five
  // blocks an SM, 147 with them and 167 without (seven at sigma_z 71: 240, 235)
  const bool many = (long long)gx.x * gx.y > 6 * 152;
#define X_ROUNDS(...)                                                                          \
  launch_x<TS, MODE, STEREO, OVER, __VA_ARGS__>(L, vin, tmp, target, conf, bounds, lambda, step,        \
                                       overwrite, halo, gx, sa, s)
  if (!STEREO && rounds <= 2) st = X_ROUNDS(STEREO ? kRoundsX : 2);
  else if (!STEREO && rounds <= 3) st = X_ROUNDS(STEREO ? kRoundsX : 3);
  else if (!STEREO && rounds <= kRoundsX && many) st = X_ROUNDS(kRoundsX, STEREO);
  else if (rounds <= kRoundsX) st = X_ROUNDS(kRoundsX);
  else st = X_ROUNDS(kRoundsWide);
#undef X_ROUNDS
  if (st) return st;
#define Y_ROWS(RM)                                                                          \
  launch_y<TS, OVER, RM>(L, tmp, vout, conf, bounds, step * lambda, overwrite, feeds, halo, \
                         gy, rows, s)
  // 8 rows a warp: twice the warps, which few tiles an SM need; 16 issue less
  // per pixel, which many do (71 against 81 us a solve of 160x120, 227 against
  // 240 us a pass over 47 Mpx); 32 where the tile has more than 256 rows (16
  // warps of 16: the registers of half an SM)
  if (rows <= 128 && px < (4 << 20)) return Y_ROWS(8);
  return rows <= 256 ? Y_ROWS(16) : Y_ROWS(32);
#undef Y_ROWS
}

template <typename TS, int MODE>
int launch_iter_t(const DtsLaunch& L, const float* vin, float* tmp, float* vout,
                  const void* target, const void* conf, const uint32_t* bounds, float lambda,
                  float step, float overwrite, int feeds, int halo, const StereoArgs* sa,
                  cudaStream_t s) {
  const StereoArgs none{nullptr, nullptr, 0.f, 0.f, 0.f, -1.f};
  const bool over = overwrite > 0.f && overwrite < 1.f;
#define ITER(ST, OV)                                                                        \
  launch_iter<TS, MODE, ST, OV>(L, vin, tmp, vout, target, conf, bounds, lambda, step,      \
                                overwrite, feeds, halo, sa ? *sa : none, s)
  if (sa) return over ? ITER(true, true) : ITER(true, false);
  return over ? ITER(false, true) : ITER(false, false);
#undef ITER
}

}  // namespace

PassGrid pass_grid(const DtsLaunch& L, int hx, int hy) {
  PassGrid G;
  for (int i = 0; i < L.n_inst; ++i) {
    const Inst& I = L.h_inst[i];
    G.rounds = std::max(G.rounds, x_rounds(I.w, I.h, x_geom(I.w, I.h, hx).halo));
    G.rows = std::max(G.rows, y_th(I.w, I.h, hy) + 2 * hy);
    G.px += (long long)I.w * I.h;
  }
  G.x = dim3(L.n_xblocks);
  G.y = dim3(L.n_yblocks);
  if (L.n_inst == 1) {
    const Inst& I = L.h_inst[0];
    const int tw = x_geom(I.w, I.h, hx).tw, th = y_th(I.w, I.h, hy);
    G.x = dim3((I.h + kXWarps - 1) / kXWarps, (I.w + tw - 1) / tw);
    G.y = dim3((I.w + 31) / 32, (I.h + th - 1) / th);
  }
  return G;
}

dim3 dts_pass_block_counts(const Inst& I, int halo) {
  const int tw = x_geom(I.w, I.h, halo).tw, th = y_th(I.w, I.h, halo);
  const unsigned xr = (I.h + kXWarps - 1) / kXWarps, xc = (I.w + tw - 1) / tw;
  const unsigned yr = (I.h + th - 1) / th, yc = (I.w + 31) / 32;
  return dim3(xr * xc, yr * yc);
}

int launch_pass_blocks(const Inst* d_inst, const Inst* h_inst, int n, int halo, Tile* x, Tile* y,
                       cudaStream_t s) {
  int nx = 0, ny = 0;
  for (int first = 0; first < n; first += kBlockStarts) {
    const int m = std::min(kBlockStarts, n - first);
    BlockStarts S = {};
    unsigned most = 1;
    for (int i = 0; i < m; ++i) {
      const dim3 c = dts_pass_block_counts(h_inst[first + i], halo);
      S.x[i] = nx;
      S.y[i] = ny;
      nx += c.x;
      ny += c.y;
      most = std::max(most, std::max(c.x, c.y));
    }
    S.x[m] = nx;
    S.y[m] = ny;
    k_pass_blocks<<<dim3((most + 255) / 256, m), 256, 0, s>>>(d_inst, first, S, halo, x, y);
    DTSGB_CUDA(cudaGetLastError());
  }
  return DTSGB_OK;
}

int launch_dts_iter(const DtsLaunch& L, Storage st, IterMode mode, const float* vin, float* tmp,
                    float* vout, const void* target, const void* conf, const uint32_t* bounds,
                    float lambda, float step, float overwrite, int feeds, int halo,
                    cudaStream_t s, const StereoArgs* stereo) {
  if (L.one_by_one()) {
    for (int i = 0; i < L.n_inst; ++i)
      if (int e = launch_dts_iter(L.one(i), st, mode, vin, tmp, vout, target, conf, bounds, lambda,
                                  step, overwrite, feeds, halo, s, stereo))
        return e;
    return DTSGB_OK;
  }
#define ITER_T(TS, M)                                                                    \
  launch_iter_t<TS, M>(L, vin, tmp, vout, target, conf, bounds, lambda, step, overwrite, \
                       feeds, halo, stereo, s)
  if (st == Storage::F32) return mode == IterMode::L2 ? ITER_T(float, 0) : ITER_T(float, 1);
  return mode == IterMode::L2 ? ITER_T(__nv_bfloat16, 0) : ITER_T(__nv_bfloat16, 1);
#undef ITER_T
}

}  // namespace dtsgb
