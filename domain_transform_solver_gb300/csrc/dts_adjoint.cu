// Adjoint of the fixed-iteration DTS solve (no reference counterpart: the
// reference has no gradients).  With the windows fixed, one iteration is
//   X: v1 = v - s*(lambda*(v - Bx v) + h(v)),  h = (c/n)(v - t)            (L2)
//                                              h = 0.5 (c/n)(v-t)/sqrt((v-t)^2+e)
//   Y: v2 = v1 - s*lambda*(v1 - By v1)
// so, for an upstream gradient g2 = dL/dv2,
//   g1 = (1 - s*lambda) g2 + s*lambda * By^T g2
//   g  = (1 - s*lambda - s*h'(v)) g1 + s*lambda * Bx^T g1
//   dL/dt += s*h'(v) g1 (and g at v_0 = t),  dL/dc += -s*(dh/dc) g1.
// B^T a at q is the sum of a(p)/n(p) over the pixels p whose window holds q.
// Each p adds its term to the interval of its window: +a at the first pixel
// of the window (clipped to the tile), -a after the last, and a prefix sum
// over the difference array gives B^T.  The terms are fixed-point integers
// (fixed_point.cuh) added with wrapping 32-bit arithmetic, so the
// shared-memory atomics that build the difference array are exact and their
// order does not matter: the result is deterministic.
// Y^T and X^T are a pass each, cut like the forward's (dts_geom.cuh).  In one
// kernel, 64 x 128 tiles with their halos in shared memory, an iteration took
// 216 us for 16 images of 1024x768 (456 instructions a pixel, two blocks an SM);
// the two passes take 146 (52 and 94), bound by issue slots and the latency of their
// loads (12 and 40 B/px).
//
// The forward iterates the adjoint needs (the X-step inputs v_k) are
// recomputed segment by segment from checkpoints v_0 = t, v_K, v_2K, ...
// saved by the forward, so memory grows with sqrt(N), not N.
#include <algorithm>

#include "../../include/dtsgb.h"
#include "dts_geom.cuh"
#include "dtsgb_internal.cuh"
#include "fixed_point.cuh"
#include "raw4.cuh"

namespace dtsgb {
namespace {

constexpr int kT = 256;
constexpr int kAdjFirst = 1, kAdjLast = 2;
// Halos above this are refused: the form before had to keep a tile and its
// halos in shared memory, and what it refused stays so (X^T is instantiated for
// up to kRoundsX rounds, which halos up to 127 need at most).
constexpr int kAdjMaxHalo = 76;

// Y^T: gout = (1 - slam) gin + slam * By^T gin.  A block per 32 columns x th
// rows, lanes on columns; a warp holds RM staged rows (gradient and bounds) in
// registers, scatters the ends of their windows into the block's difference
// array (lanes on 32 banks) and completes the rows of the tile among them.
template <int RM>
__global__ void __launch_bounds__(RM == 32 ? 768 : 512, RM == 8 ? 3 : RM == 16 ? 2 : 1)
    k_adj_y(const Inst* __restrict__ insts, const float* __restrict__ gin,
            float* __restrict__ gout, const uint32_t* __restrict__ bnd, float slam, int hy,
            const Tile* __restrict__ blocks) {
  extern __shared__ unsigned smy[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = blockDim.x;
  const Tile t = blocks ? blocks[blockIdx.x] : Tile{0, (int)blockIdx.x, (int)blockIdx.y, 0};
  const Inst in = insts[t.inst];
  const int W = in.w, H = in.h, P = in.pitch;
  const int th = y_th(W, H, hy), rows = th + 2 * hy, warps = rows / RM;
  const int nrt = 2 * hy + 2;
  unsigned* smax = smy;
  float* rtab = reinterpret_cast<float*>(smy + 1);  // 1/n
  unsigned* tot = smy + 1 + nrt;                    // warps x 32
  unsigned* D = tot + warps * 32;                   // (rows + 1) x 32
  for (int i = tid; i < nrt; i += nt) rtab[i] = i ? __frcp_rn((float)i) : 0.f;
  for (int i = tid; i < (rows + 1) * 32; i += nt) D[i] = 0u;
  if (tid == 0) *smax = 0u;
  __syncthreads();
  pdl_wait_then_release();
  if (warp >= warps) return;  // (whole warps; see the barriers)
  const int live = 32 * warps;
  const int x = t.x0 * 32 + lane, y0 = t.y0 * th;
  const bool inx = x < W;
  const int s0 = warp * RM;      // the warp's first staged row
  const int ys = y0 - hy + s0;   // its image row
  const long long first = in.off + (long long)ys * P + x;
  const float* gc = gin + first;
  const uint32_t* bc = bnd + first;
  float v[RM];
  uint32_t b[RM];
  if (t.x0 * 32 + 32 <= W && ys >= 0 && ys + RM <= H) {  // the whole warp inside
#pragma unroll
    for (int k = 0; k < RM; ++k) v[k] = __ldg(gc + (long long)k * P);
#pragma unroll
    for (int k = 0; k < RM; ++k) b[k] = __ldg(bc + (long long)k * P) >> 16;
  } else {
#pragma unroll
    for (int k = 0; k < RM; ++k) {
      const bool ok = inx && (unsigned)(ys + k) < (unsigned)H;
      v[k] = ok ? __ldg(gc + (long long)k * P) : 0.f;
      b[k] = ok ? __ldg(bc + (long long)k * P) >> 16 : 0u;
    }
  }
  float m = 0.f;
#pragma unroll
  for (int k = 0; k < RM; ++k) m = fmaxf(m, fabsf(v[k] * rtab[window_count(b[k], hy)]));
  m = warp_max_nonneg(m);
  if (lane == 0) atomicMax(smax, __float_as_uint(m));
  asm volatile("bar.sync 1, %0;" ::"r"(live) : "memory");
  const int F = fx_shift(__uint_as_float(*smax), ceil_log2(2 * hy + 1));
  const float sF = pow2f(F), isF = pow2f(-F);
#pragma unroll
  for (int k = 0; k < RM; ++k) {
    if (b[k]) {  // (a window holds its pixel: 0 is outside the image)
      const int dl = (int)(b[k] & 0xff), du = (int)(b[k] >> 8);
      const unsigned A = fx_from(v[k] * rtab[window_count(b[k], hy)], sF);
      atomicAdd(D + max(s0 + k - dl + 1, 0) * 32 + lane, A);
      atomicAdd(D + min(s0 + k + du + 1, rows) * 32 + lane, 0u - A);
    }
  }
  asm volatile("bar.sync 1, %0;" ::"r"(live) : "memory");
  const unsigned* Dw = D + s0 * 32 + lane;
  unsigned acc = 0u;
#pragma unroll
  for (int k = 0; k < RM; ++k) acc += Dw[k * 32];
  tot[warp * 32 + lane] = acc;
  asm volatile("bar.sync 1, %0;" ::"r"(live) : "memory");
  if (!inx) return;
  acc = 0u;
  for (int w = 0; w < warp; ++w) acc += tot[w * 32 + lane];
  const int k0 = max(hy - s0, 0), k1 = min(min(th, H - y0) + hy - s0, RM);  // tile rows
  float* oc = gout + first;
#pragma unroll
  for (int k = 0; k < RM; ++k) {
    acc += Dw[k * 32];
    if (k >= k0 && k < k1)
      oc[(long long)k * P] = __fmaf_rn(1.f - slam, v[k], slam * fx_window(acc, 0u, isF));
  }
}

// X^T and the parameter gradients, from g1 = Y^T's result: a warp per row
// segment, four adjacent pixels a lane and round in registers, the difference
// array and its prefix in the warp's shared memory.  Gradients may differ by
// orders of magnitude along a row, so a segment whose 32-column cells do (by
// more than 4 bits in their largest terms, for windows of up to 32 pixels; by
// less for wider ones, whose conversions weigh more) is summed cell by cell,
// each with a fixed-point scale of its own: a term goes, in its scale, to each
// cell that its window reaches.  With one scale for up to 512 columns 20 large
// gradients in 400x300 small ones took the median error of the small from
// 2e-7 to 4.5e-6 (6e-7 so); all segments cell by cell cost 25% of a training
// step, those that need it 1%.  flags: kAdjFirst, the
// first adjoint of a backward (dL/dt and dL/dc start at zero: not read);
// kAdjLast, the last (its dL/dv_0 goes into dL/dt, as v_0 = t, instead of to
// gout).  The five planes of a round are loaded when the round is due: loads a
// round ahead held 124 registers, four blocks an SM (115 us against 90).
template <typename TS, int MODE, int NR>
__global__ void __launch_bounds__(32 * kXWarps, 7)
    k_adj_x(const Inst* __restrict__ insts, const float* __restrict__ g1p,
            float* __restrict__ gout, const float* __restrict__ vk, const TS* __restrict__ tgt,
            const TS* __restrict__ cnf, const uint32_t* __restrict__ bnd,
            float* __restrict__ grad_t, float* __restrict__ grad_c, float lambda, float step,
            int hx, int flags, const Tile* __restrict__ blocks) {
  using PX = XPrefix<NR>;
  extern __shared__ unsigned smx[];
  const bool read = !(flags & kAdjFirst), last = flags & kAdjLast;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned* S = smx + warp * (4 * PX::QS);
  char* Sb = reinterpret_cast<char*>(S);
  float* qmax = reinterpret_cast<float*>(smx + kXWarps * 4 * PX::QS) + warp * (36 * NR);
  int* cellF = reinterpret_cast<int*>(qmax + 32 * NR);  // the cells' scales
  float* rtab = reinterpret_cast<float*>(smx + kXWarps * (4 * PX::QS + 36 * NR));  // 1/n
  const Tile t = blocks ? blocks[blockIdx.x] : Tile{0, (int)blockIdx.y, (int)blockIdx.x, 0};
  const Inst in = insts[t.inst];
  const int W = in.w;
  const XGeom g = x_geom(W, in.h, hx);
  const int row = t.y0 * kXWarps + warp, x0 = t.x0 * g.tw;
  const int nrt = 2 * hx + 2;
  for (int i = tid; i < nrt; i += 32 * kXWarps) rtab[i] = i ? __frcp_rn((float)i) : 0.f;
#pragma unroll
  for (int r = 0; r < NR; ++r)
#pragma unroll
    for (int k = 0; k < 4; ++k) S[k * PX::QS + lane + 32 * r] = 0u;
  __syncthreads();
  pdl_wait_then_release();
  if (row >= in.h) return;
  const int xe = min(x0 + g.tw, W);
  const int rounds = (xe - x0 + g.halo + 127) >> 7;
  const int xl = x0 - g.ha + 4 * lane;  // the lane's first pixel of round 0
  const long long base = in.off + (long long)row * in.pitch;
  float4 v[NR];
  uint4 b[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const int x = xl + 128 * r;
    v[r] = make_float4(0.f, 0.f, 0.f, 0.f);
    b[r] = make_uint4(0u, 0u, 0u, 0u);
    if (x >= 0 && x < W && r < rounds) {
      v[r] = __ldg(reinterpret_cast<const float4*>(g1p + base + x));
      b[r] = __ldg(reinterpret_cast<const uint4*>(bnd + base + x));
      // columns past the width: the pitch's padding
      if (x + 1 >= W) b[r].y = 0u;
      if (x + 2 >= W) b[r].z = 0u;
      if (x + 3 >= W) b[r].w = 0u;
    }
  }
  struct Quad {
    float4 v, gt, gc;
    Raw4<TS> tv, cv;
  };
  auto mine = [&](int r) { return xl + 128 * r >= x0 && xl + 128 * r < xe; };
  auto fetch = [&](int r, Quad& Q) {
    if (r < rounds && mine(r)) {
      const long long p = base + xl + 128 * r;
      Q.v = __ldg(reinterpret_cast<const float4*>(vk + p));
      Q.tv.load(tgt + p);
      Q.cv.load(cnf + p);
      if (read) {
        Q.gt = *reinterpret_cast<const float4*>(grad_t + p);
        Q.gc = *reinterpret_cast<const float4*>(grad_c + p);
      }
    }
  };
  Quad Q;
  Q.v = Q.gt = Q.gc = make_float4(0.f, 0.f, 0.f, 0.f);
  Q.tv.zero();
  Q.cv.zero();
  // n of a pixel of its packed bounds (0 outside the image: 1/n = 0)
  auto count = [hx](uint32_t w) { return window_count(w, hx); };
  // the largest term of the segment, and the smallest of its cells' largest
  // (cells of zeros aside)
  const int lgx = ceil_log2(2 * hx + 1);
  unsigned most = 0u, least = ~0u;
#pragma unroll
  for (int r = 0; r < NR; ++r)
    if (r < rounds) {
      float m = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        m = fmaxf(m, fabsf(f4_get(v[r], k) * rtab[count(u4_get(b[r], k))]));
      unsigned c = __float_as_uint(m);
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) c = max(c, __shfl_xor_sync(0xffffffffu, c, o));
      most = max(most, c);
      least = min(least, c - 1u);  // (zero: the largest)
    }
  most = __reduce_max_sync(0xffffffffu, most);
  least = __reduce_min_sync(0xffffffffu, least) + 1u;
  const bool cells = (int)(most >> 23) - (int)(least >> 23) > max(9 - lgx, 0);
  // 2^F for sums of 2hx + 1 terms up to m (their conversions' halves are within
  // the 1.0001)
  auto scale = [&](unsigned bits) {
    const float m = __uint_as_float(bits), sum = 1.0001f * (float)(2 * hx + 1) * m;
    return sum <= 3.4e38f ? fx_shift(sum, 0) : fx_shift(m, lgx);
  };
  const int F = scale(most);
  float isF = pow2f(-F);
  if (!cells) {
    const float sF = pow2f(F);
    const int end = 128 * rounds;
#pragma unroll
    for (int r = 0; r < NR; ++r)
      if (r < rounds)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t w = u4_get(b[r], k);
          if (w) {
            const int dl = (int)(w & 0xff), du = (int)((w >> 8) & 0xff);
            const int i = 4 * lane + 128 * r + k;
            const unsigned A = fx_from(f4_get(v[r], k) * rtab[count(w)], sF);
            atomicAdd(PX::entry(Sb, max(i - dl + 1, 0)), A);
            atomicAdd(PX::entry(Sb, min(i + du + 1, end)), 0u - A);
          }
        }
  } else {
    // a cell's scale: from the terms whose windows may reach it
#pragma unroll
    for (int r = 0; r < NR; ++r)
      if (r < rounds) {
        float m = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          m = fmaxf(m, fabsf(f4_get(v[r], k) * rtab[count(u4_get(b[r], k))]));
        qmax[lane + 32 * r] = m;
      }
    __syncwarp();
    const int reach = (hx + 3) >> 2;  // in quads
    for (int r = 0; r < rounds; ++r) {
      const int q0 = (lane & 24) + 32 * r;  // the cell's first quad
      unsigned m = 0u;
      for (int j = (lane & 7) - reach; j < 8 + reach; j += 8)
        m = max(m, __float_as_uint(qmax[min(max(q0 + j, 0), 32 * rounds - 1)]));
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
      if ((lane & 7) == 0) cellF[(lane >> 3) + 4 * r] = scale(m);
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < NR; ++r)
      if (r < rounds) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t w = u4_get(b[r], k);
          if (w) {
            const int dl = (int)(w & 0xff), du = (int)((w >> 8) & 0xff);
            const int i = 4 * lane + 128 * r + k;
            const int a = max(i - dl + 1, 0), e = i + du + 1;  // the window: [a, e)
            const float term = f4_get(v[r], k) * rtab[count(w)];
            for (int c = a >> 5; c < 4 * rounds && 32 * c < e; ++c) {
              const unsigned A = fx_from(term, pow2f(cellF[c]));
              atomicAdd(PX::entry(Sb, max(a, 32 * c)), A);
              if (e < 32 * c + 32) atomicAdd(PX::entry(Sb, e), 0u - A);
            }
          }
        }
      }
  }
  __syncwarp();
  const float slam = step * lambda;
  unsigned carry = 0u;
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    if (r < rounds) {
      unsigned a[4];
      fetch(r, Q);
#pragma unroll
      for (int k = 0; k < 4; ++k) a[k] = S[k * PX::QS + lane + 32 * r];
#pragma unroll
      for (int k = 1; k < 4; ++k) a[k] += a[k - 1];
      unsigned off;
      if (cells) {
        off = a[3];  // of the cell's lanes up to this one
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
          const unsigned n = __shfl_up_sync(0xffffffffu, off, o, 8);
          if ((lane & 7) >= o) off += n;
        }
        off -= a[3];
        isF = pow2f(-cellF[(lane >> 3) + 4 * r]);
      } else {
        const unsigned incl = warp_incl_scan(a[3], lane);
        off = carry + incl - a[3];
        carry += __shfl_sync(0xffffffffu, incl, 31);
      }
      const Quad& q = Q;
      if (!mine(r)) continue;
      float go[4], gt[4], gc[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float bt = fx_window(off + a[k], 0u, isF);
        const float g1 = f4_get(v[r], k), rn = rtab[count(u4_get(b[r], k))];
        const float vv = f4_get(q.v, k), tv = q.tv[k], cv = q.cv[k];
        const float d = vv - tv;
        float dh_dv, dh_dc;
        if (MODE == 0) {
          dh_dv = cv * rn;
          dh_dc = d * rn;
        } else {
          const float rt = __fsqrt_rn(__fmaf_rn(d, d, 1e-6f));
          dh_dv = __fdiv_rn(0.5f * (cv * rn) * 1e-6f, rt * rt * rt);
          dh_dc = __fdiv_rn(0.5f * d * rn, rt);
        }
        go[k] = __fmaf_rn(1.f - slam - step * dh_dv, g1, slam * bt);
        gt[k] = f4_get(q.gt, k) + step * dh_dv * g1;
        gc[k] = f4_get(q.gc, k) - step * dh_dc * g1;
        if (last) gt[k] += go[k];
      }
      const int x = xl + 128 * r;
      const long long p = base + x;
      if (x + 4 <= W) {
        if (!last) *reinterpret_cast<float4*>(gout + p) = make_float4(go[0], go[1], go[2], go[3]);
        *reinterpret_cast<float4*>(grad_t + p) = make_float4(gt[0], gt[1], gt[2], gt[3]);
        *reinterpret_cast<float4*>(grad_c + p) = make_float4(gc[0], gc[1], gc[2], gc[3]);
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (x + k < W) {
            if (!last) gout[p + k] = go[k];
            grad_t[p + k] = gt[k];
            grad_c[p + k] = gc[k];
          }
      }
    }
  }
}

__global__ void k_axpy_planes(const Inst* __restrict__ insts, const float* __restrict__ a,
                              float* __restrict__ y) {
  const Inst in = insts[blockIdx.y];
  const long long n = (long long)in.pitch * in.h;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[in.off + i] += a[in.off + i];
}

template <int RM>
int launch_y(const DtsLaunch& L, const PassGrid& G, const float* gin, float* gout,
             const uint32_t* bounds, float slam, int hy, cudaStream_t s) {
  auto kern = k_adj_y<RM>;
  const int warps = G.rows / RM;
  const size_t smem = sizeof(unsigned) *
                      ((size_t)(2 * hy + 3) + warps * 32 + ((size_t)G.rows + 1) * 32);
  DTSGB_CUDA(allow_smem(kern, smem));
  ProfScope ps(s, DTSGB_K_DTS_ADJOINT);
  DTSGB_CUDA(launch_dependent(kern, G.y, dim3(32 * warps), smem, s, L.d_inst, gin, gout, bounds,
                              slam, hy, L.n_inst > 1 ? L.d_yblocks : (const Tile*)nullptr));
  return DTSGB_OK;
}

template <typename TS, int MODE>
int launch_adj_t(const DtsLaunch& L, float* g, float* g1, const float* vk, const void* t,
                 const void* c, const uint32_t* bounds, float* gt, float* gc, float lambda,
                 float step, int halo, int flags, cudaStream_t s) {
  const PassGrid G = pass_grid(L, halo, halo);
  const float slam = step * lambda;
  int st;
  // the rows a warp holds: as the forward's Y pass
  if (G.rows <= 128 && G.px < (4 << 20)) st = launch_y<8>(L, G, g, g1, bounds, slam, halo, s);
  else if (G.rows <= 256) st = launch_y<16>(L, G, g, g1, bounds, slam, halo, s);
  else st = launch_y<32>(L, G, g, g1, bounds, slam, halo, s);
  if (st) return st;
  auto x = [&](auto kern, int nr, int qs) -> int {
    const size_t smem = sizeof(unsigned) * ((size_t)kXWarps * (4 * qs + 36 * nr) + 2 * halo + 2);
    ProfScope ps(s, DTSGB_K_DTS_ADJOINT);
    DTSGB_CUDA(launch_dependent(kern, G.x, dim3(32 * kXWarps), smem, s, L.d_inst, g1, g, vk,
                                (const TS*)t, (const TS*)c, bounds, gt, gc, lambda, step, halo,
                                flags, L.n_inst > 1 ? L.d_xblocks : (const Tile*)nullptr));
    return DTSGB_OK;
  };
  if (G.rounds <= 2) return x(k_adj_x<TS, MODE, 2>, 2, XPrefix<2>::QS);
  if (G.rounds <= 3) return x(k_adj_x<TS, MODE, 3>, 3, XPrefix<3>::QS);
  return x(k_adj_x<TS, MODE, kRoundsX>, kRoundsX, XPrefix<kRoundsX>::QS);
}

// One iteration's adjoint of g, in place (g1: scratch).
int launch_adjoint(const DtsLaunch& L, Storage st, IterMode mode, float* g, float* g1,
                   const float* vk, const void* t, const void* c, const uint32_t* bounds,
                   float* gt, float* gc, float lambda, float step, int halo, int flags,
                   cudaStream_t s) {
  if (L.one_by_one()) {
    for (int i = 0; i < L.n_inst; ++i)
      if (int e = launch_adjoint(L.one(i), st, mode, g, g1, vk, t, c, bounds, gt, gc, lambda, step,
                                 halo, flags, s))
        return e;
    return DTSGB_OK;
  }
#define ADJ_T(TS, M) \
  launch_adj_t<TS, M>(L, g, g1, vk, t, c, bounds, gt, gc, lambda, step, halo, flags, s)
  if (st == Storage::F32) return mode == IterMode::L2 ? ADJ_T(float, 0) : ADJ_T(float, 1);
  return mode == IterMode::L2 ? ADJ_T(__nv_bfloat16, 0) : ADJ_T(__nv_bfloat16, 1);
#undef ADJ_T
}

}  // namespace

int dts_checkpoint_segment(int num_iterations) {
  // fewest planes held (ceil(N/K) - 1 + K), and among those the fewest
  // recomputed iterations (N - ceil(N/K)): the smallest such K
  const int n = std::max(num_iterations, 1);
  int best = 1;
  long long best_planes = -1;
  for (int k = 1; k <= n; ++k) {
    const long long planes = (n + k - 1) / k - 1 + k;
    if (best_planes < 0 || planes < best_planes) {
      best_planes = planes;
      best = k;
    }
  }
  return best;
}

int dts_forward_checkpointed(const DtsLaunch& L, Storage st, IterMode mode,
                             const DtsGrad& G, const void* target, const void* conf,
                             const uint32_t* bounds, float lambda, float step, int halo,
                             int num_iterations, float* v0, float* v1, cudaStream_t s) {
  if (num_iterations <= 0) return launch_init_var(L, st, target, v0, s);
  const float* cur = nullptr;
  int st_ = first_iterate(L, st, target, v0, &cur, s);
  if (st_) return st_;
  for (int next = 1; next <= num_iterations; ++next) {
    float* dst = next < num_iterations && next % G.seg == 0 ? G.cp[next / G.seg - 1] : v0;
    st_ = launch_dts_iter(L, st, mode, cur, v1, dst, target, conf, bounds, lambda, step, -1.f, 0,
                          halo, s);
    if (st_) return st_;
    cur = dst;
  }
  return DTSGB_OK;
}

int dts_backward(const DtsLaunch& L, const Inst* d_inst, int n_inst, long long plane,
                 Storage st, IterMode mode, const DtsGrad& G, const void* target,
                 const void* conf, const uint32_t* bounds, float lambda, float step,
                 int halo, int num_iterations, float* tmp, float* grad_t, float* grad_c,
                 cudaStream_t s) {
  if (num_iterations <= 0) {  // v = t: dL/dt = dL/dv, dL/dc = 0
    DTSGB_CUDA(cudaMemsetAsync(grad_t, 0, plane * sizeof(float), s));
    DTSGB_CUDA(cudaMemsetAsync(grad_c, 0, plane * sizeof(float), s));
    k_axpy_planes<<<dim3(64, n_inst), kT, 0, s>>>(d_inst, G.g[0], grad_t);
    DTSGB_CUDA(cudaGetLastError());
    return DTSGB_OK;
  }
  // the first adjoint writes dL/dt and dL/dc (no zeroing pass), the last
  // adds dL/dv_0 to dL/dt (no final pass)
  if (halo > kAdjMaxHalo)
    return fail(DTSGB_ERR_UNSUPPORTED, "sigma_z too large for the adjoint");
  const int nseg = (num_iterations + G.seg - 1) / G.seg;
  for (int j = nseg - 1; j >= 0; --j) {
    const int start = j * G.seg;
    const int len = std::min(G.seg, num_iterations - start);
    // X-step inputs v_start .. v_start+len-1 of this segment: the first is
    // t (segment 0) or a checkpoint, the others are recomputed into segbuf
    const float* x0 = nullptr;
    if (j > 0) {
      x0 = G.cp[j - 1];
    } else if (int st_ = first_iterate(L, st, target, G.segbuf[0], &x0, s)) {
      return st_;
    }
    for (int k = 1; k < len; ++k) {
      int st_ = launch_dts_iter(L, st, mode, k == 1 ? x0 : G.segbuf[k - 1], tmp, G.segbuf[k],
                                target, conf, bounds, lambda, step, -1.f, 0, halo, s);
      if (st_) return st_;
    }
    for (int k = len - 1; k >= 0; --k) {
      const int flags = (j == nseg - 1 && k == len - 1 ? kAdjFirst : 0) |
                        (j == 0 && k == 0 ? kAdjLast : 0);
      // (G.g[0] holds dL/dv_N on entry)
      int st_ = launch_adjoint(L, st, mode, G.g[0], G.g[1], k == 0 ? x0 : G.segbuf[k], target,
                               conf, bounds, grad_t, grad_c, lambda, step, halo, flags, s);
      if (st_) return st_;
    }
  }
  return DTSGB_OK;
}

}  // namespace dtsgb
