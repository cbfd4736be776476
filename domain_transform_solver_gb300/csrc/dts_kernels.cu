// DTS kernels for sm_103a: guide ingest, the domain-transform filter pass with
// the confidence epilogue, and small helpers for downloads.  The window bounds
// are in dts_bounds.cu, the iteration in dts_passes.cu.
//
// Key fact used throughout: the edge weights dH, dV are >= 1
// (sqrt(1 + nonnegative)), so a window of the reference's linear search
// (src/domain_transform_filter.cuh:7-28) never reaches further than
// floor(sigma)+1 pixels from its centre.  Every pass is therefore a
// bounded-radius stencil (here over tiles plus halo in shared memory, in
// dts_passes.cu over segments of a row or strips of columns): no global prefix
// sums, no transposes, no long-row cancellation.
#include <algorithm>
#include <cmath>

#include "../../include/dtsgb.h"
#include "color.cuh"
#include "dtsgb_internal.cuh"
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

}  // namespace

int launch_color_convert_flat(uchar4* guide, long long n, int color_space,
                              cudaStream_t s) {
  if (color_space == DTSGB_RGB || n <= 0) return DTSGB_OK;
  k_color_convert_flat<<<grid_for(n), kThreads, 0, s>>>(guide, n, color_space);
  DTSGB_CUDA(cudaGetLastError());
  return DTSGB_OK;
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
  DTSGB_CUDA((allow_smem(k_filter<NCH, CONF, TS, TW, TH>, smem)));
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
