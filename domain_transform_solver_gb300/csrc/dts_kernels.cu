// DTS kernels for sm_103a: guide ingest, window-bound search, the
// domain-transform filter pass with the confidence epilogue, and small helpers
// for downloads.  The iteration is in dts_passes.cu.
//
// Key fact used throughout: the edge weights dH, dV are >= 1
// (sqrt(1 + nonnegative)), so a window of the reference's linear search
// (src/domain_transform_filter.cuh:7-28) never reaches further than
// floor(sigma)+1 pixels from its centre.  Every pass is therefore a
// bounded-radius stencil over a tile plus halo held in shared memory: no
// global prefix sums, no transposes, no long-row cancellation.
#include <algorithm>
#include <cmath>

#include "../../include/dtsgb.h"
#include "color.cuh"
#include "dtsgb_internal.cuh"
#include "fixed_point.cuh"
#include "raw4.cuh"

namespace dtsgb {

namespace {

constexpr int kThreads = 256;

__global__ void k_color_convert_flat(uchar4* __restrict__ g, long long n,
                                     int cs) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    g[i] = convert_pixel(g[i], cs);
}

// ---------------------------------------------------------------------------
// Window bounds (a4).  One CTA per TWxTH tile, 256 threads.
// Lower bound: the largest i < p with sum_{j=i+1..p} w(j) > sigma, else p-1.
// Upper bound: (the smallest i > p, i < limit, with sum_{j=p+1..i} w(j) >
// sigma) - 1, else p.  limit is W for X and min(W,H) (reference quirk) or H
// for Y.  A negative ratio stands for an all-zero domain transform (no
// differential computed yet): every window is the pixel itself.
//
// The weights are clamped to sigma + 1 (a window holding a larger one
// exceeds sigma either way) and converted to fixed point at 2^F with
// r * (sigma + 1) * 2^F <= 2^30, so a window sum is the exact difference of
// two wrapping 32-bit prefixes of the converted weights (each within 2^-F-1
// of the float weight: decisions differ from float sums only within about
// r * 2^-F of the threshold).  Shared memory holds the prefix of dH along
// each tile row over [x0 - r, x0 + TW + r) and of dV along each tile column
// over [y0 - r, y0 + TH + r).  As p moves forward, both window ends move
// forward, so a thread walks a segment of 8 pixels with two pointers that
// only advance: about two prefix reads per end and pixel instead of a search
// over the whole radius.
// ---------------------------------------------------------------------------
// Pixels per thread and axis of the two-pointer walks (a launch knob:
// DTSGB_TUNE_BOUNDS_SEGMENT selects 4, 8 or 16).
constexpr int kBoundsSegDefault = 8;

// Lower and upper window ends along one axis for the n pixels starting at
// prefix index j0 (S[j0 + k] for pixel p0 + k), coordinates p0.., axis length
// `len` (lower limit 0), upper limit `lim`; stride between prefix entries s.
// Writes dl | du << 8 to out[k * os].
__device__ __forceinline__ void bounds_walk(const unsigned* __restrict__ S, int s, int j0,
                                            int p0, int n, int r, int lim, int T,
                                            uint16_t* out, int os) {
  int q = 0, u = 0;
  for (int k = 0; k < n; ++k) {
    const int j = j0 + k, p = p0 + k;
    const unsigned Sj = S[j * s];
    // lower: the largest q in [j - K, j - 1] with S[j] - S[q] > T (K = min(r, p)),
    // advanced from the previous pixel's (both only move forward)
    const int qmin = j - min(r, p);
    q = k == 0 ? qmin - 1 : max(q, qmin - 1);
    while (q + 1 <= j - 1 && (int)(Sj - S[(q + 1) * s]) > T) ++q;
    const int dl = q >= qmin ? j - q : 1;
    // upper: the smallest u in [j + 1, j + K'] with S[u] - S[j] > T
    // (K' = min(r, lim - 1 - p)); the first pixel starts from the far end
    const int umax = j + min(r, lim - 1 - p);
    if (k == 0) {
      u = umax + 1;
      while (u - 1 > j && (int)(S[(u - 1) * s] - Sj) > T) --u;
    } else {
      u = max(u, j + 1);
      while (u <= umax && (int)(S[u * s] - Sj) <= T) ++u;
    }
    const int du = u <= umax ? u - j - 1 : 0;
    out[k * os] = (uint16_t)(dl | (du << 8));
  }
}

template <int TW, int TH, int SEG>
__global__ void __launch_bounds__(kThreads)
    k_bounds(const Inst* __restrict__ insts, const Tile* __restrict__ tiles,
             const uchar4* __restrict__ guide, uint32_t* __restrict__ bounds,
             float ratio_x, float ratio_y, int rx, int ry, int ref_y_limit,
             float cap_x, float cap_y, float scale_x, float scale_y, int Tx, int Ty) {
  static_assert(TW == 32 && TH == 32 && kThreads == 256, "bounds tile shape");
  static_assert(SEG == 4 || SEG == 8 || SEG == 16, "walk segment");
  constexpr int NW = kThreads / 32;
  extern __shared__ unsigned smu[];
  const Tile t = tiles[blockIdx.x];
  const Inst in = insts[t.inst];
  const int W = in.w, H = in.h, P = in.pitch;
  const uchar4* g = guide + in.off;
  const int DW = TW + 2 * rx, DWp = DW | 1;  // odd row stride: lanes on rows
  const int DR = TH + 2 * ry;
  unsigned* SH = smu;             // TH x DWp: prefix of dH, entry 0 = 0 at x0 - rx
  unsigned* SV = SH + TH * DWp;   // DR x TW: prefix of dV, entry 0 = 0 at y0 - ry
  uint16_t* BX = reinterpret_cast<uint16_t*>(SV + DR * TW);  // TH x TW
  uint16_t* BY = BX + TH * TW;                               // TH x TW
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // ---- 1. weights in fixed point.  dH: a warp per row, lanes on columns; a
  // lane's left neighbour comes from the lane before it (one load per pixel).
  // dV: eight threads per column, each down a run of rows, the pixel above
  // carried in a register.  Pixels outside the image read as zero.
  auto load_g = [&](int x, int y) -> unsigned {
    return (x >= 0 && x < W && y >= 0 && y < H)
               ? *reinterpret_cast<const unsigned*>(g + (long long)y * P + x)
               : 0u;
  };
  auto as_px = [](unsigned v) { return *reinterpret_cast<const uchar4*>(&v); };
  for (int r = warp; r < TH; r += NW) {
    const int y = t.y0 + r;
    for (int j0 = 0; j0 < DW; j0 += 32) {
      const int j = j0 + lane, x = t.x0 - rx + j;
      const unsigned cur = j < DW ? load_g(x, y) : 0u;
      unsigned prev = __shfl_up_sync(0xffffffffu, cur, 1);
      if (lane == 0) prev = load_g(x - 1, y);
      unsigned q = 0u;
      if (j > 0 && x >= 0 && x < W && y < H && ratio_x >= 0.f)
        q = (unsigned)__float2int_rn(
            fminf(edge_weight(as_px(cur), as_px(prev), ratio_x), cap_x) * scale_x);
      if (j < DW) SH[r * DWp + j] = q;
    }
  }
  {
    const int c = tid % TW, sgi = tid / TW, nsg = kThreads / TW;
    const int seg = (DR + nsg - 1) / nsg;
    const int j0 = sgi * seg, j1 = min(DR, j0 + seg);
    const int x = t.x0 + c;
    unsigned prev = load_g(x, t.y0 - ry + j0 - 1);
    for (int j = j0; j < j1; ++j) {
      const int y = t.y0 - ry + j;
      const unsigned cur = load_g(x, y);
      unsigned q = 0u;
      if (j > 0 && x < W && y >= 0 && y < H && ratio_y >= 0.f)
        q = (unsigned)__float2int_rn(
            fminf(edge_weight(as_px(cur), as_px(prev), ratio_y), cap_y) * scale_y);
      SV[j * TW + c] = q;
      prev = cur;
    }
  }
  __syncthreads();
  // ---- 2. inclusive prefixes: a thread per row of SH, a thread per column of SV
  // (a segmented scan over all warps was slower: its extra pass costs more
  // issue slots than the serial chains, which the other resident blocks hide)
  if (tid < TH) {
    unsigned* row = SH + tid * DWp;
    unsigned acc = 0u;
    for (int j = 0; j < DW; ++j) row[j] = acc += row[j];
  } else if (tid >= 32 && tid < 32 + TW) {
    unsigned* col = SV + (tid - 32);
    unsigned acc = 0u;
    for (int j = 0; j < DR; ++j) col[j * TW] = acc += col[j * TW];
  }
  __syncthreads();
  // ---- 3. two-pointer walks: warps 0-3 rows (X), warps 4-7 columns (Y), each
  // taking the SEG-pixel segments sg = warp, warp + 4, ... of its lines
  const int ylim = ref_y_limit ? min(W, H) : H;
  constexpr int NSEG = TW / SEG;
  if (tid < 4 * 32) {
    const int r = lane, y = t.y0 + r;  // lanes on rows
    for (int sg = warp; sg < NSEG; sg += 4) {
      const int xs = t.x0 + sg * SEG;
      const int n = min(SEG, W - xs);
      if (y < H && n > 0)
        bounds_walk(SH + r * DWp, 1, xs - t.x0 + rx, xs, n, rx, W, Tx,
                    BX + r * TW + sg * SEG, 1);
    }
  } else {
    const int c = lane, x = t.x0 + c;  // lanes on columns
    for (int sg = warp - 4; sg < NSEG; sg += 4) {
      const int ys = t.y0 + sg * SEG;
      const int n = min(SEG, H - ys);
      if (x < W && n > 0)
        bounds_walk(SV + c, TW, ys - t.y0 + ry, ys, n, ry, ylim, Ty, BY + sg * SEG * TW + c,
                    TW);
    }
  }
  __syncthreads();
  // ---- 4. packed bounds, rows written coalesced
  uint32_t* bo = bounds + in.off;
  for (int i = tid; i < TH * TW; i += kThreads) {
    const int r = i / TW, c = i % TW;
    const int x = t.x0 + c, y = t.y0 + r;
    if (x < W && y < H) bo[y * P + x] = (uint32_t)BX[i] | ((uint32_t)BY[i] << 16);
  }
}

// ---------------------------------------------------------------------------
// Filter pass (a5): X box mean then Y box mean over NCH channels sharing the
// windows (src/domain_transform_filter.cuh:30-71).  With CONF the Y result
// is not stored; instead the confidence epilogue of
// src/domain_transform_solver.cu:21-44 is applied to (ch0, ch1) =
// (DT(t), DT(t^2)).
// ---------------------------------------------------------------------------
template <int NCH, bool CONF, typename TS, int TW, int TH>
__global__ void __launch_bounds__(kThreads)
    k_filter(const Inst* __restrict__ insts, const Tile* __restrict__ tiles,
             const float* __restrict__ in0, const float* __restrict__ in1,
             float* __restrict__ out0, float* __restrict__ out1,
             const uint32_t* __restrict__ bnd, int hx, int hy,
             TS* __restrict__ conf_out, float scale, int left_clear) {
  extern __shared__ float sm[];
  const Tile t = tiles[blockIdx.x];
  const Inst in = insts[t.inst];
  const int W = in.w, H = in.h, P = in.pitch;
  const long long off = in.off;
  const int SW = TW + 2 * hx, SR = TH + 2 * hy;
  float* sv[NCH];
  float* sx[NCH];
  for (int ch = 0; ch < NCH; ++ch) {
    sv[ch] = sm + ch * (SR * SW + SR * TW);
    sx[ch] = sv[ch] + SR * SW;
  }
  const float* src[2] = {in0, in1};
  const int gx0 = t.x0 - hx, gy0 = t.y0 - hy;
  for (int i = threadIdx.x; i < SR * SW; i += blockDim.x) {
    const int r = i / SW, c = i - r * SW;
    const int x = gx0 + c, y = gy0 + r;
    const bool ok = x >= 0 && x < W && y >= 0 && y < H;
    const long long p = off + (long long)y * P + x;
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) sv[ch][i] = ok ? __ldg(src[ch] + p) : 0.f;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < SR * TW; i += blockDim.x) {
    const int r = i / TW, c = i - r * TW;
    const int x = t.x0 + c, y = gy0 + r;
    float res[NCH];
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) res[ch] = 0.f;
    if (x < W && y >= 0 && y < H) {
      const long long p = off + (long long)y * P + x;
      const uint32_t b = __ldg(bnd + p);
      // radii clamped to the staged halo: a window never reads outside it
      const int dl = min((int)(b & 0xff), hx + 1), du = min((int)((b >> 8) & 0xff), hx);
      const float nf = (float)(dl + du);
#pragma unroll
      for (int ch = 0; ch < NCH; ++ch) {
        const float* row = sv[ch] + r * SW + (c + hx);
        float s = 0.f;
        for (int k = 1 - dl; k <= du; ++k) s += row[k];
        res[ch] = __fdiv_rn(s, nf);
      }
    }
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) sx[ch][i] = res[ch];
  }
  __syncthreads();
  float* dst[2] = {out0, out1};
  for (int i = threadIdx.x; i < TH * TW; i += blockDim.x) {
    const int r = i / TW, c = i - r * TW;
    const int x = t.x0 + c, y = t.y0 + r;
    if (x >= W || y >= H) continue;
    const long long p = off + (long long)y * P + x;
    const uint32_t b = __ldg(bnd + p);
    const int dl = min((int)((b >> 16) & 0xff), hy + 1), du = min((int)(b >> 24), hy);
    const float nf = (float)(dl + du);
    float res[NCH];
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) {
      const float* col = sx[ch] + (r + hy) * TW + c;
      float s = 0.f;
      for (int k = 1 - dl; k <= du; ++k) s += col[k * TW];
      res[ch] = __fdiv_rn(s, nf);
    }
    if (CONF) {
      float cv = 0.f;
      if (x > left_clear) {
        const float var = res[1] - res[0] * res[0];
        cv = (var < 0.f || !isfinite(var)) ? 0.f : expf(-var * scale);
      }
      conf_out[p] = store_cast<TS>(cv);
      // keep DT(t^2) as the filter's last result (the reference leaves it in
      // its var buffer)
      dst[1][p] = res[1];
      dst[0][p] = res[0];
    } else {
#pragma unroll
      for (int ch = 0; ch < NCH; ++ch) dst[ch][p] = res[ch];
    }
  }
}

// Storage plane -> float plane (and its square): four elements per thread and
// 16-byte accesses (rows are pitched to 32 elements, so an instance is a
// whole number of aligned groups).
template <typename TS>
__global__ void k_to_float(const Inst* __restrict__ insts, const TS* __restrict__ src,
                           float* __restrict__ dst, float* __restrict__ dst_sq) {
  const Inst in = insts[blockIdx.y];
  const long long n = (long long)in.pitch * in.h;
  for (long long i = 4 * (blockIdx.x * (long long)blockDim.x + threadIdx.x); i < n;
       i += 4 * (long long)gridDim.x * blockDim.x) {
    Raw4<TS> v;
    v.load(src + in.off + i);
    *reinterpret_cast<float4*>(dst + in.off + i) = make_float4(v[0], v[1], v[2], v[3]);
    if (dst_sq)
      *reinterpret_cast<float4*>(dst_sq + in.off + i) =
          make_float4(v[0] * v[0], v[1] * v[1], v[2] * v[2], v[3] * v[3]);
  }
}

template <typename TS>
__global__ void k_from_float(const float* __restrict__ src, TS* __restrict__ dst,
                             long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    dst[i] = store_cast<TS>(src[i]);
}

template <typename TS>
__global__ void k_fill(TS* __restrict__ dst, long long n, float v) {
  const TS val = store_cast<TS>(v);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    dst[i] = val;
}

__global__ void k_differential(const Inst* __restrict__ insts,
                               const uchar4* __restrict__ guide, float ratio,
                               int axis, float* __restrict__ out) {
  const Inst in = insts[blockIdx.y];
  const long long n = (long long)in.w * in.h;
  const uchar4 zero = make_uchar4(0, 0, 0, 0);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int y = (int)(i / in.w), x = (int)(i - (long long)y * in.w);
    const long long p = in.off + (long long)y * in.pitch + x;
    const uchar4 cur = guide[p];
    uchar4 prev = zero;
    if (axis == 0 && x > 0) prev = guide[p - 1];
    if (axis == 1 && y > 0) prev = guide[p - in.pitch];
    out[p] = edge_weight(cur, prev, ratio);
  }
}

// Row-wise inclusive prefix sum, one warp per row, Kahan-compensated carry
// between 32-element chunks.
__global__ void k_row_prefix(const Inst* __restrict__ insts,
                             const float* __restrict__ in,
                             float* __restrict__ out) {
  const Inst I = insts[blockIdx.y];
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= I.h) return;
  const float* src = in + I.off + (long long)warp * I.pitch;
  float* dst = out + I.off + (long long)warp * I.pitch;
  float carry = 0.f, comp = 0.f;
  for (int x0 = 0; x0 < I.w; x0 += 32) {
    const int x = x0 + lane;
    float v = x < I.w ? src[x] : 0.f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float n = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += n;
    }
    if (x < I.w) dst[x] = carry + v;
    const float total = __shfl_sync(0xffffffffu, v, 31);
    const float yk = total - comp;
    const float tk = carry + yk;
    comp = (tk - carry) - yk;
    carry = tk;
  }
}

__global__ void k_unpack_bounds(const Inst* __restrict__ insts,
                                const uint32_t* __restrict__ bnd, int axis,
                                int32_t* __restrict__ l, int32_t* __restrict__ u) {
  const Inst in = insts[blockIdx.y];
  const long long n = (long long)in.w * in.h;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int y = (int)(i / in.w), x = (int)(i - (long long)y * in.w);
    const uint32_t b = bnd[in.off + (long long)y * in.pitch + x];
    const int pos = axis == 0 ? x : y;
    const int dl = axis == 0 ? (b & 0xff) : ((b >> 16) & 0xff);
    const int du = axis == 0 ? ((b >> 8) & 0xff) : (b >> 24);
    l[i] = pos - dl;
    u[i] = pos + du;
  }
}

int grid_for(long long n, int threads = kThreads) {
  long long b = (n + threads - 1) / threads;
  if (b > 152 * 16) b = 152 * 16;
  if (b < 1) b = 1;
  return (int)b;
}

template <typename F>
int set_smem(F* f, size_t bytes) {
  if (bytes > 48 * 1024) {
    DTSGB_CUDA(cudaFuncSetAttribute(
        f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  }
  return DTSGB_OK;
}

constexpr size_t kMaxSmem = 227 * 1024;

}  // namespace

int launch_color_convert_flat(uchar4* guide, long long n, int color_space,
                              cudaStream_t s) {
  if (color_space == DTSGB_RGB || n <= 0) return DTSGB_OK;
  k_color_convert_flat<<<grid_for(n), kThreads, 0, s>>>(guide, n, color_space);
  DTSGB_CUDA(cudaGetLastError());
  return DTSGB_OK;
}

int launch_bounds(const DtsLaunch& L, const uchar4* guide, uint32_t* bounds,
                  float ratio_x, float ratio_y, float sigma_x, float sigma_y,
                  int ref_y_limit, cudaStream_t s) {
  const int rx = (int)floorf(sigma_x) + 1, ry = (int)floorf(sigma_y) + 1;
  if (rx > 255 || ry > 255)
    return fail(DTSGB_ERR_UNSUPPORTED, "sigma >= 255 is not supported");
  const int TW = kBoundsTW, TH = kBoundsTH;
  const size_t smem = sizeof(unsigned) * ((size_t)TH * ((TW + 2 * rx) | 1) +
                                          (size_t)(TH + 2 * ry) * TW) +
                      2 * sizeof(uint16_t) * TH * TW;
  if (smem > kMaxSmem) return fail(DTSGB_ERR_UNSUPPORTED, "sigma too large");
  // fixed point per axis: r * (sigma + 1) * 2^F <= 2^30; threshold floor(sigma 2^F)
  auto fx = [](int r, float sigma, float* cap, float* scale, int* T) {
    *cap = sigma + 1.f;
    const int F = 30 - (int)std::ceil(std::log2((double)r * (double)*cap));
    *scale = std::ldexp(1.f, F);
    *T = (int)std::floor((double)sigma * std::ldexp(1.0, F));
  };
  float cap_x, cap_y, scale_x, scale_y;
  int Tx, Ty;
  fx(rx, sigma_x, &cap_x, &scale_x, &Tx);
  fx(ry, sigma_y, &cap_y, &scale_y, &Ty);
  auto go = [&](auto kern) -> int {
    int st = set_smem(kern, smem);
    if (st) return st;
    ProfScope ps(s, DTSGB_K_BOUNDS);
    kern<<<L.n_tiles, kThreads, smem, s>>>(L.d_inst, L.d_tiles, guide, bounds, ratio_x,
                                           ratio_y, rx, ry, ref_y_limit, cap_x, cap_y,
                                           scale_x, scale_y, Tx, Ty);
    DTSGB_CUDA(cudaGetLastError());
    return DTSGB_OK;
  };
  if (L.bounds_seg == 4) return go(k_bounds<kBoundsTW, kBoundsTH, 4>);
  if (L.bounds_seg == 16) return go(k_bounds<kBoundsTW, kBoundsTH, 16>);
  return go(k_bounds<kBoundsTW, kBoundsTH, kBoundsSegDefault>);
}

int launch_target_to_float(const DtsLaunch& L, Storage st, const void* src,
                           float* dst, float* dst_sq, cudaStream_t s) {
  // enough blocks for the largest instance (64 left most SMs idle on one image)
  long long most = 1 << 20;
  if (L.h_inst) {
    most = 1;
    for (int i = 0; i < L.n_inst; ++i)
      most = std::max(most, (long long)L.h_inst[i].pitch * L.h_inst[i].h);
  }
  const int cap = std::max(64, 152 * 16 / L.n_inst);
  const dim3 grid(std::min(grid_for((most + 3) / 4), cap), L.n_inst);
  ProfScope ps(s, DTSGB_K_DTS_OTHER);
  if (st == Storage::F32)
    k_to_float<float><<<grid, kThreads, 0, s>>>(L.d_inst, (const float*)src, dst, dst_sq);
  else
    k_to_float<__nv_bfloat16><<<grid, kThreads, 0, s>>>(
        L.d_inst, (const __nv_bfloat16*)src, dst, dst_sq);
  DTSGB_CUDA(cudaGetLastError());
  return DTSGB_OK;
}

int launch_init_var(const DtsLaunch& L, Storage st, const void* target,
                    float* v, cudaStream_t s) {
  return launch_target_to_float(L, st, target, v, nullptr, s);
}

int first_iterate(const DtsLaunch& L, Storage st, const void* target, float* v,
                  const float** first, cudaStream_t s) {
  *first = st == Storage::F32 ? static_cast<const float*>(target) : v;
  return st == Storage::F32 ? DTSGB_OK : launch_init_var(L, st, target, v, s);
}

int launch_storage_from_float(const Inst*, int, Storage st, const float* src,
                              void* dst, long long n, cudaStream_t s) {
  if (st == Storage::F32) {
    DTSGB_CUDA(cudaMemcpyAsync(dst, src, n * sizeof(float),
                               cudaMemcpyDeviceToDevice, s));
    return DTSGB_OK;
  }
  k_from_float<__nv_bfloat16><<<grid_for(n), kThreads, 0, s>>>(
      src, (__nv_bfloat16*)dst, n);
  DTSGB_CUDA(cudaGetLastError());
  return DTSGB_OK;
}

int launch_fill_storage(Storage st, void* dst, long long n, float value,
                        cudaStream_t s) {
  if (st == Storage::F32)
    k_fill<float><<<grid_for(n), kThreads, 0, s>>>((float*)dst, n, value);
  else
    k_fill<__nv_bfloat16><<<grid_for(n), kThreads, 0, s>>>(
        (__nv_bfloat16*)dst, n, value);
  DTSGB_CUDA(cudaGetLastError());
  return DTSGB_OK;
}

template <int NCH, bool CONF, typename TS, int TW, int TH>
static int launch_filter_shape(const DtsLaunch& L, const float* in0,
                               const float* in1, float* out0, float* out1,
                               const uint32_t* bounds, int hx, int hy,
                               void* conf_out, float scale, int left_clear,
                               cudaStream_t s) {
  const size_t smem = NCH * sizeof(float) *
                      ((size_t)(TH + 2 * hy) * (TW + 2 * hx) + (size_t)(TH + 2 * hy) * TW);
  if (smem > kMaxSmem) return fail(DTSGB_ERR_UNSUPPORTED, "filter sigma too large");
  int st = set_smem(k_filter<NCH, CONF, TS, TW, TH>, smem);
  if (st) return st;
  ProfScope ps(s, DTSGB_K_FILTER);
  k_filter<NCH, CONF, TS, TW, TH><<<L.n_tiles, kThreads, smem, s>>>(
      L.d_inst, L.d_tiles, in0, in1, out0, out1, bounds, hx, hy, (TS*)conf_out,
      scale, left_clear);
  DTSGB_CUDA(cudaGetLastError());
  return DTSGB_OK;
}

template <int NCH, bool CONF, typename TS>
static int launch_filter_t(const DtsLaunch& L, const float* in0,
                           const float* in1, float* out0, float* out1,
                           const uint32_t* bounds, int hx, int hy,
                           void* conf_out, float scale, int left_clear,
                           cudaStream_t s) {
  if (L.small)
    return launch_filter_shape<NCH, CONF, TS, kIterSmallTW, kIterSmallTH>(
        L, in0, in1, out0, out1, bounds, hx, hy, conf_out, scale, left_clear, s);
  if (L.d_tiles_small &&
      NCH * sizeof(float) * ((size_t)(kIterTH + 2 * hy) * (kIterTW + 2 * hx) +
                             (size_t)(kIterTH + 2 * hy) * kIterTW) > kMaxSmem)
    return launch_filter_shape<NCH, CONF, TS, kIterSmallTW, kIterSmallTH>(
        L.as_small(), in0, in1, out0, out1, bounds, hx, hy, conf_out, scale, left_clear, s);
  return launch_filter_shape<NCH, CONF, TS, kIterTW, kIterTH>(
      L, in0, in1, out0, out1, bounds, hx, hy, conf_out, scale, left_clear, s);
}

int launch_filter_pass(const DtsLaunch& L, int nch, const float* in0,
                       const float* in1, float* out0, float* out1,
                       const uint32_t* bounds, int hx, int hy, Storage st,
                       void* conf_out, float scale, int left_clear,
                       cudaStream_t s) {
  if (conf_out) {
    if (st == Storage::F32)
      return launch_filter_t<2, true, float>(L, in0, in1, out0, out1, bounds, hx,
                                             hy, conf_out, scale, left_clear, s);
    return launch_filter_t<2, true, __nv_bfloat16>(L, in0, in1, out0, out1,
                                                   bounds, hx, hy, conf_out,
                                                   scale, left_clear, s);
  }
  if (nch == 2)
    return launch_filter_t<2, false, float>(L, in0, in1, out0, out1, bounds, hx,
                                            hy, nullptr, 0.f, 0, s);
  return launch_filter_t<1, false, float>(L, in0, nullptr, out0, nullptr, bounds,
                                          hx, hy, nullptr, 0.f, 0, s);
}

int launch_differential(const DtsLaunch& L, const uchar4* guide, float ratio,
                        int axis, float* out, cudaStream_t s) {
  k_differential<<<dim3(64, L.n_inst), kThreads, 0, s>>>(L.d_inst, guide, ratio,
                                                         axis, out);
  DTSGB_CUDA(cudaGetLastError());
  return DTSGB_OK;
}

int launch_row_prefix(const Inst* h_inst, const Inst* d_inst, int n_inst,
                      const float* in, float* out, cudaStream_t s) {
  int max_h = 1;
  for (int i = 0; i < n_inst; ++i) max_h = max_h > h_inst[i].h ? max_h : h_inst[i].h;
  const int warps_per_block = kThreads / 32;
  dim3 grid((max_h + warps_per_block - 1) / warps_per_block, n_inst);
  k_row_prefix<<<grid, kThreads, 0, s>>>(d_inst, in, out);
  DTSGB_CUDA(cudaGetLastError());
  return DTSGB_OK;
}

int launch_unpack_bounds(const DtsLaunch& L, const uint32_t* bounds, int axis,
                         int32_t* l, int32_t* u, cudaStream_t s) {
  k_unpack_bounds<<<dim3(64, L.n_inst), kThreads, 0, s>>>(L.d_inst, bounds, axis,
                                                          l, u);
  DTSGB_CUDA(cudaGetLastError());
  return DTSGB_OK;
}

}  // namespace dtsgb
