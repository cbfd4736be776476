// HFBS kernels for sm_103a (Mazumdar et al. bilateral-grid solver as the
// reference implements it, src/hfbs.cu:65-427).
//
// Every kernel handles a batch of independent instances: blockIdx.y selects
// the instance, blockIdx.x strides over its pixels / voxels / lines (CTAs
// past the end of a small instance exit at once).  Grids are dense
// gx*gy*gl float arrays, x fastest.  Reads outside the interior follow the
// reference's buffers (see hfbs_internal.cuh / the oracle): index -1 reads 0
// (zero boundary mode), index g reads the pad value of that buffer.
//
// The splat is atomic-free and deterministic: the threads of a spatial cell
// bin its pixels into per-thread luma histograms held in shared memory.
#include <algorithm>
#include <vector>

#include "../../include/dtsgb.h"
#include "dtsgb_internal.cuh"
#include "fixed_point.cuh"
#include "hfbs_internal.cuh"
#include "tma.cuh"

namespace dtsgb {

namespace {

constexpr int kT = 256;

__device__ __forceinline__ long long gidx(const HInst& I, int x, int y, int z) {
  return I.grid_off + ((long long)z * I.gy + y) * I.px + x;
}

// a12: SplatBAndC + BistochastasizeSetup (src/hfbs.cu:72-120).  Bins
// (floor(x/sx), floor(y/sy), floor(L/sl)) with L the .x channel; sums of
// c*t, c and 1 per bin.  Luma bin == gl lands in the overflow plane.
template <typename TS>
__global__ void __launch_bounds__(64)
    k_splat(const HInst* __restrict__ insts, const uchar4* __restrict__ guide,
            const TS* __restrict__ tgt, const TS* __restrict__ cnf,
            float* __restrict__ count, float* __restrict__ csum,
            float* __restrict__ b, float* __restrict__ ovf, HParams p) {
  extern __shared__ float sh[];
  __shared__ int lbin[256];  // luma bin of each 8-bit luma value
  const HInst I = insts[blockIdx.y];
  const int ncell = I.gx * I.gy;
  const int cell = blockIdx.x * blockDim.x + threadIdx.x;
  const int gl = I.gl;
  // per-thread histograms: [bin][3] strided by blockDim for conflict-free use
  float* hist = sh;
  const int T = blockDim.x;
  if (blockIdx.x * blockDim.x >= ncell) return;
  for (int l = threadIdx.x; l < 256; l += T)
    lbin[l] = (int)floorf((float)l * 1.0f / p.sigma_l);
  __syncthreads();
  for (int k = 0; k < 3 * gl; ++k) hist[k * T + threadIdx.x] = 0.f;
  float ovf_cnt = 0.f;
  if (cell < ncell) {
    const int bx = cell % I.gx, by = cell / I.gx;
    const int xs = cell_start(bx, p.sigma_x, I.w), xe = cell_start(bx + 1, p.sigma_x, I.w);
    const int ys = cell_start(by, p.sigma_y, I.h), ye = cell_start(by + 1, p.sigma_y, I.h);
    // a run of pixels in the same luma bin is summed in registers and added
    // to the cell's histogram when the bin changes (a fixed order: the
    // result is deterministic)
    int run = -1;
    float r_ct = 0.f, r_c = 0.f, r_n = 0.f;
    auto flush = [&]() {
      if (run < 0) return;
      if (run < gl) {
        hist[(3 * run + 0) * T + threadIdx.x] += r_ct;
        hist[(3 * run + 1) * T + threadIdx.x] += r_c;
        hist[(3 * run + 2) * T + threadIdx.x] += r_n;
      } else {
        ovf_cnt += r_n;
      }
    };
    constexpr int U = 8;  // pixels whose loads are issued together
    for (int y = ys; y < ye; ++y) {
      const long long row = I.pix_off + (long long)y * I.pitch;
      for (int x0 = xs; x0 < xe; x0 += U) {
        int lum[U];
        float cv[U], tv[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
          lum[k] = 0;
          cv[k] = tv[k] = 0.f;
          if (x0 + k < xe) {
            lum[k] = guide[row + x0 + k].x;
            cv[k] = load_f(cnf + row + x0 + k);
            tv[k] = load_f(tgt + row + x0 + k);
          }
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
          if (x0 + k >= xe) break;
          const int bl = lbin[lum[k]];
          const float ct = __fmul_rn(cv[k], tv[k]);  // (not fused: as k_splat_cell)
          if (bl != run) {
            flush();
            run = bl;
            r_ct = ct;
            r_c = cv[k];
            r_n = 1.f;
          } else {
            r_ct = __fadd_rn(r_ct, ct);
            r_c += cv[k];
            r_n += 1.f;
          }
        }
      }
    }
    flush();
    for (int z = 0; z < gl; ++z) {
      const long long gi = gidx(I, bx, by, z);
      b[gi] = hist[(3 * z + 0) * T + threadIdx.x];
      csum[gi] = hist[(3 * z + 1) * T + threadIdx.x];
      count[gi] = hist[(3 * z + 2) * T + threadIdx.x];
    }
    ovf[I.plane_off + cell] = I.ovf_stored ? ovf_cnt : 0.f;
  }
}

// a12 for large cells: a CTA per cell, bit for bit k_splat's sums.  Those
// are sums in row-major order of the cell's runs (neighbours in one luma
// bin), each run summed in order first, so the work a thread of k_splat
// does alone splits into parallel parts that keep every addition: the
// pixels of a chunk are loaded together into shared memory, run starts are
// found and compacted by a block scan, runs are summed by a thread each, and
// a thread per luma bin adds the runs of its bin in order.  The run that a
// chunk ends in stays open into the next one.  From kSplatCellPx pixels a
// cell on: one thread a cell took 850 us for the 374 cells of 64 x 64
// pixels of a 1376x1088 image (latency of one batch of loads after the
// other, 6 CTAs); at 8 x 8 pixels the thread per cell is the faster one.
constexpr int kSplatCellPx = 256;
constexpr int kSplatChunk = 1024, kSplatCellT = 256, kSplatPer = kSplatChunk / kSplatCellT;

template <typename TS>
__global__ void __launch_bounds__(kSplatCellT)
    k_splat_cell(const HInst* __restrict__ insts, const uchar4* __restrict__ guide,
                 const TS* __restrict__ tgt, const TS* __restrict__ cnf,
                 float* __restrict__ count, float* __restrict__ csum, float* __restrict__ b,
                 float* __restrict__ ovf, HParams p) {
  constexpr int T = kSplatCellT, NW = T / 32;
  __shared__ int lbin[256];                      // luma bin of each 8-bit luma value
  __shared__ short sbin[kSplatChunk];            // the chunk's pixels: bin, c, c*t
  __shared__ float sc[kSplatChunk], sct[kSplatChunk];
  __shared__ short rs[kSplatChunk], rb[kSplatChunk];  // its runs: start, bin, sums
  __shared__ float rct[kSplatChunk], rc[kSplatChunk], rn[kSplatChunk];
  __shared__ int wsum[NW];
  __shared__ int o_bin;                          // the open run (-1: none)
  __shared__ float o_ct, o_c, o_n;
  const HInst I = insts[blockIdx.y];
  const int cell = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (cell >= I.gx * I.gy) return;
  const int gl = I.gl;
  if (tid < 256) lbin[tid] = (int)floorf((float)tid * 1.0f / p.sigma_l);
  if (tid == 0) o_bin = -1;
  const int bx = cell % I.gx, by = cell / I.gx;
  const int xs = cell_start(bx, p.sigma_x, I.w), xe = cell_start(bx + 1, p.sigma_x, I.w);
  const int ys = cell_start(by, p.sigma_y, I.h), ye = cell_start(by + 1, p.sigma_y, I.h);
  const int nx = xe - xs, total = nx * (ye - ys);
  float h_ct = 0.f, h_c = 0.f, h_n = 0.f;  // bin tid's sums
  __syncthreads();
  for (int base = 0; base < total; base += kSplatChunk) {
    const int n = min(kSplatChunk, total - base);
    unsigned char lum[kSplatPer];
    float cv[kSplatPer], tv[kSplatPer];
#pragma unroll
    for (int j = 0; j < kSplatPer; ++j) {
      const int i = min(tid + j * T, n - 1) + base;
      const int y = i / nx, x = i - y * nx;
      const long long g = I.pix_off + (long long)(ys + y) * I.pitch + xs + x;
      lum[j] = guide[g].x;
      cv[j] = load_f(cnf + g);
      tv[j] = load_f(tgt + g);
    }
#pragma unroll
    for (int j = 0; j < kSplatPer; ++j) {
      const int i = tid + j * T;
      if (i < n) {
        sbin[i] = (short)lbin[lum[j]];
        sc[i] = cv[j];
        sct[i] = __fmul_rn(cv[j], tv[j]);
      }
    }
    __syncthreads();
    // run starts among this thread's kSplatPer neighbours, compacted in order
    const int open = o_bin, i0 = tid * kSplatPer;
    int prev = i0 == 0 ? open : (i0 <= n ? sbin[i0 - 1] : 0), starts = 0, k = 0;
#pragma unroll
    for (int j = 0; j < kSplatPer; ++j) {
      if (i0 + j < n) {
        const int c = sbin[i0 + j];
        if (c != prev) starts |= 1 << j;
        prev = c;
      }
    }
    const int mine = __popc(starts);
    const int incl = (int)warp_incl_scan((unsigned)mine, lane);
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int R = 0;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      if (w < warp) k += wsum[w];
      R += wsum[w];
    }
    k += incl - mine;
#pragma unroll
    for (int j = 0; j < kSplatPer; ++j)
      if (starts >> j & 1) rs[k++] = (short)(i0 + j);
    __syncthreads();
    // a thread per run; the last thread extends the open run to the first start
    for (int r = tid; r < R; r += T) {
      const int a = rs[r], e = r + 1 < R ? rs[r + 1] : n;
      float u = sct[a], v = sc[a], m = 1.f;
      for (int i = a + 1; i < e; ++i) {
        u += sct[i];
        v += sc[i];
        m += 1.f;
      }
      rb[r] = sbin[a];
      rct[r] = u;
      rc[r] = v;
      rn[r] = m;
    }
    if (tid == T - 1 && open >= 0) {
      const int e = R > 0 ? rs[0] : n;
      float u = o_ct, v = o_c, m = o_n;
      for (int i = 0; i < e; ++i) {
        u += sct[i];
        v += sc[i];
        m += 1.f;
      }
      o_ct = u;
      o_c = v;
      o_n = m;
    }
    __syncthreads();
    // a thread per bin (bin gl: the overflow count) adds its closed runs
    if (R > 0) {
      if (tid <= gl) {
        if (open == tid) {
          h_ct += o_ct;
          h_c += o_c;
          h_n += o_n;
        }
#pragma unroll 4
        for (int r = 0; r + 1 < R; ++r)
          if (rb[r] == tid) {
            h_ct += rct[r];
            h_c += rc[r];
            h_n += rn[r];
          }
      }
      __syncthreads();
      if (tid == 0) {
        o_bin = rb[R - 1];
        o_ct = rct[R - 1];
        o_c = rc[R - 1];
        o_n = rn[R - 1];
      }
    }
    __syncthreads();
  }
  if (tid <= gl && o_bin == tid) {
    h_ct += o_ct;
    h_c += o_c;
    h_n += o_n;
  }
  if (tid < gl) {
    const long long gi = gidx(I, bx, by, tid);
    b[gi] = h_ct;
    csum[gi] = h_c;
    count[gi] = h_n;
  } else if (tid == gl) {
    ovf[I.plane_off + cell] = I.ovf_stored ? h_n : 0.f;
  }
}

// The elementwise kernels below run flat over the whole grid arena: the
// voxels in the gaps between instances are computed too and never read.
__global__ void k_fill_ones(float* __restrict__ a, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    a[i] = 1.f;
}

// a13: one BistochastasizeOptimize step (src/hfbs.cu:126-155):
// n' = sqrt(n * (count + 1e-5) / (2n + sum6 nbr n + 1e-5)).  Faces covered by
// FillGrid read `pad`, all other out-of-grid reads 0.
__global__ void k_bistoch(const HInst* __restrict__ insts,
                          const float* __restrict__ src, float* __restrict__ dst,
                          const float* __restrict__ count, float pad) {
  pdl_wait_then_release();  // launched as a dependent of the previous pass
  const HInst I = insts[blockIdx.y];
  const int gx = I.gx, gy = I.gy, gl = I.gl;
  const float px = I.cov_x ? pad : 0.f, py = I.cov_y ? pad : 0.f,
              pz = I.cov_l ? pad : 0.f;
  const float* s = src + I.grid_off;
  const float* cn = count + I.grid_off;
  float* d = dst + I.grid_off;
  const int sy = I.px, sz = I.px * gy;
  // one thread per (x, y) column, marching along l: the l-neighbours come
  // from registers, and the loads of level l+1 are issued before level l is
  // computed
  for (int cl = blockIdx.x * blockDim.x + threadIdx.x; cl < gx * gy;
       cl += gridDim.x * blockDim.x) {
    const int y = cl / gx, x = cl - y * gx;
    const int col = y * sy + x;
    const bool xm = x > 0, xp = x + 1 < gx, ym = y > 0, yp = y + 1 < gy;
    auto nb4 = [&](int i, float (&o)[5]) {  // x-1, x+1, y-1, y+1, count
      o[0] = xm ? s[i - 1] : 0.f;
      o[1] = xp ? s[i + 1] : px;
      o[2] = ym ? s[i - sy] : 0.f;
      o[3] = yp ? s[i + sy] : py;
      o[4] = cn[i];
    };
    float vprev = 0.f, vcur = s[col];
    float cur[5], nxt[5];
    nb4(col, cur);
    for (int l = 0; l < gl; ++l) {
      const int i = l * sz + col;
      const bool more = l + 1 < gl;
      const float vnext = more ? s[i + sz] : pz;
      if (more) nb4(i + sz, nxt);
      float a = cur[0];
      a += cur[1];
      a += cur[2];
      a += cur[3];
      a += l > 0 ? vprev : 0.f;
      a += vnext;
      const float blurred = 2.f * vcur + a;
      d[i] = __fsqrt_rn(__fdiv_rn(vcur * (cur[4] + 0.00001f), blurred + 0.00001f));
      vprev = vcur;
      vcur = vnext;
#pragma unroll
      for (int k = 0; k < 5; ++k) cur[k] = nxt[k];
    }
  }
}

// a14: CalcInvDiagA (src/hfbs.cu:159-195):
// invA = 1 / max(1e-3, lambda*(count - 2 n^2) + sum c), evaluated by the
// reference in double and stored as float.  For a float d, rounding 1/d to
// double and then to float gives the correctly rounded float reciprocal (a
// product of a 24-bit and a 25-bit significand cannot come within 2^-53 of 1
// without equalling it, so 1/d never lands within a double ulp of a float
// midpoint), so the FP64 division is replaced by __frcp_rn.  d >= 1e-3f is
// the float form of (double)d > 1e-3, and 1/1e-3 rounds to 1000 (NaN too,
// as fmax returns the other operand).
__global__ void k_inv_diag(const float* __restrict__ count, const float* __restrict__ csum,
                           const float* __restrict__ norm, float* __restrict__ invA,
                           float lambda, long long n) {
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < n;
       g += (long long)gridDim.x * blockDim.x) {
    const float nv = norm[g];
    const float diag = lambda * (count[g] - 2.f * nv * nv) + csum[g];
    invA[g] = diag >= 1e-3f ? __frcp_rn(diag) : 1000.f;
  }
}

// a15 along x (contiguous lines): one warp per line.  The forward recursion
// F(i) = s(i) + beta*F(i-1) and the backward one S(i) = s(i) + beta*S(i+1)
// are decayed scans over 32-element chunks (Hillis-Steele with beta^o weights,
// carry scaled by beta^(lane+1) between chunks); d(i) = F(i) + beta*S(i+1).
__global__ void k_laplace_x(const HInst* __restrict__ insts,
                            const float* __restrict__ s0, float* __restrict__ d0,
                            const float* __restrict__ s1, float* __restrict__ d1,
                            float beta) {
  const HInst I = insts[blockIdx.y];
  const int gx = I.gx, nlines = I.gy * I.gl;
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  float bo[5];  // beta^1, beta^2, beta^4, beta^8, beta^16
  bo[0] = beta;
#pragma unroll
  for (int k = 1; k < 5; ++k) bo[k] = bo[k - 1] * bo[k - 1];
  float blane = 1.f;  // beta^(lane+1)
  for (int k = 0; k <= lane; ++k) blane *= beta;
  float brev = 1.f;  // beta^(32-lane)
  for (int k = lane; k < 32; ++k) brev *= beta;
  for (int line = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; line < nlines;
       line += nwarps) {
    const long long base = I.grid_off + (long long)line * I.px;
    for (int f = blockIdx.z; f < 2; f += gridDim.z) {  // the field
      const float* s = (f ? s1 : s0) + base;
      float* d = (f ? d1 : d0) + base;
      // forward: F
      float carry = 0.f;
      for (int x0 = 0; x0 < gx; x0 += 32) {
        const int x = x0 + lane;
        float r = x < gx ? s[x] : 0.f;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
          const float t = __shfl_up_sync(0xffffffffu, r, 1 << k);
          if (lane >= (1 << k)) r = __fmaf_rn(bo[k], t, r);
        }
        r = __fmaf_rn(blane, carry, r);
        if (x < gx) d[x] = r;
        carry = __shfl_sync(0xffffffffu, r, 31);
      }
      // backward: S over reversed chunks, add beta * S(i+1)
      carry = 0.f;  // S of the first element after the chunk
      const int last0 = ((gx - 1) / 32) * 32;
      for (int x0 = last0; x0 >= 0; x0 -= 32) {
        const int x = x0 + lane;
        float r = x < gx ? s[x] : 0.f;  // suffix scan runs from lane 31 down
#pragma unroll
        for (int k = 0; k < 5; ++k) {
          const float t = __shfl_down_sync(0xffffffffu, r, 1 << k);
          if (lane + (1 << k) < 32) r = __fmaf_rn(bo[k], t, r);
        }
        // lanes past the end hold zeros, so the suffix needs no masking;
        // add the carried S of the next chunk, decayed by beta^(32-lane)
        r = __fmaf_rn(brev, carry, r);
        float next = __shfl_down_sync(0xffffffffu, r, 1);  // S(i+1)
        if (lane == 31) next = carry;
        if (x < gx) d[x] = __fmaf_rn(beta, next, d[x]);
        carry = __shfl_sync(0xffffffffu, r, 0);
      }
    }
  }
}

// a15: Laplace sweep along one axis for two fields at once (src/hfbs.cu:
// 355-427): d(i) = sum_j beta^|i-j| s(j), forward then backward recursion,
// one thread per grid line (used along y and l, where consecutive threads
// take consecutive x and the accesses coalesce).  The recursions are serial,
// their loads are not: each thread loads kLapChunk elements of a line before
// it runs the recursion over them, so that a chunk's loads are in flight
// together instead of one load latency per element.
constexpr int kLapChunk = 8;
__global__ void k_laplace(const HInst* __restrict__ insts, int axis,
                          const float* __restrict__ s0, float* __restrict__ d0,
                          const float* __restrict__ s1, float* __restrict__ d1,
                          float beta) {
  const int f = blockIdx.z;  // the field: a line of each is a thread's work
  constexpr int U = kLapChunk;
  const HInst I = insts[blockIdx.y];
  const int gx = I.gx, gy = I.gy, gl = I.gl;
  int len, na, nlines;
  long long stride;
  const int px = I.px;
  if (axis == 1) {
    len = gy; stride = px; na = gx; nlines = gx * gl;
  } else {
    len = gl; stride = (long long)px * gy; na = gx; nlines = gx * gy;
  }
  for (int line = blockIdx.x * blockDim.x + threadIdx.x; line < nlines;
       line += gridDim.x * blockDim.x) {
    const int a = line % na, bb = line / na;
    long long base;
    if (axis == 1) base = (long long)bb * px * gy + a;
    else base = (long long)bb * px + a;
    base += I.grid_off;
    {
      const float* s = (f ? s1 : s0) + base;
      float* d = (f ? d1 : d0) + base;
      // forward: d(0) = s(0), d(i) = beta * d(i-1) + s(i)
      float r = 0.f;
      for (int i0 = 0; i0 < len; i0 += U) {
        float v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = i0 + u < len ? s[(i0 + u) * stride] : 0.f;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int i = i0 + u;
          if (i < len) {
            r = i == 0 ? v[u] : __fmaf_rn(beta, r, v[u]);
            d[i * stride] = r;
          }
        }
      }
      // backward: r(len-1) = s(len-1); for i < len-1: r = beta * r,
      // d(i) += r, r += s(i)
      r = s[(long long)(len - 1) * stride];
      for (int i0 = len - 2; i0 >= 0; i0 -= U) {
        float v[U], w[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int i = i0 - u;
          v[u] = i >= 0 ? s[i * stride] : 0.f;
          w[u] = i >= 0 ? d[i * stride] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int i = i0 - u;
          if (i >= 0) {
            r = beta * r;
            d[i * stride] = w[u] + r;
            r = r + v[u];
          }
        }
      }
    }
  }
}

// The same along l for grids of up to NL levels: a line stays in registers, so
// each element is read and written once (the general form reads it twice more
// and writes it once more; at 64 levels it is the faster one, 73 against 102 us
// on 408 x 306).
template <int NL>
__global__ void __launch_bounds__(128)
    k_laplace_l(const HInst* __restrict__ insts, const float* __restrict__ s0,
                float* __restrict__ d0, const float* __restrict__ s1, float* __restrict__ d1,
                float beta) {
  const HInst I = insts[blockIdx.y];
  const int px = I.px, gl = I.gl;
  const float* sf = (blockIdx.z ? s1 : s0) + I.grid_off;
  float* df = (blockIdx.z ? d1 : d0) + I.grid_off;
  const int plane = px * I.gy;  // (the padding columns too: they are never read)
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < plane; c += gridDim.x * blockDim.x) {
    float v[NL], w[NL];
#pragma unroll
    for (int l = 0; l < NL; ++l) v[l] = l < gl ? sf[(long long)l * plane + c] : 0.f;
    float r = 0.f;
#pragma unroll
    for (int l = 0; l < NL; ++l) w[l] = r = l == 0 ? v[0] : __fmaf_rn(beta, r, v[l]);
    r = 0.f;
#pragma unroll
    for (int l = NL - 1; l >= 0; --l) {
      if (l + 1 < gl) w[l] = __fmaf_rn(beta, r, w[l]);
      if (l < gl) r = l + 1 < gl ? __fmaf_rn(beta, r, v[l]) : v[l];
    }
#pragma unroll
    for (int l = 0; l < NL; ++l)
      if (l < gl) df[(long long)l * plane + c] = w[l];
  }
}

// (float)((double)b / ((double)c + 1e-7)) without double arithmetic, which
// is slow on this part.  The denominator c + 1e-7 is carried as floats
// dh + dl to about 2^-48 of itself: an exact two-sum of c and the float
// nearest 1e-7, plus the rest of the double 1e-7.  q0 = b / dh is correctly
// rounded, so b - q0 * dh is exact by FMA, and q0 + (b - q0 * d) / dh carries
// the quotient to about 2^-46 of itself before the final rounding: it can
// differ from the double quotient's rounding only when that lies within
// about 2^-22 ulp of a float rounding midpoint.
__device__ __forceinline__ float div_by_c_plus_eps(float b, float c) {
  constexpr float e_hi = 1e-7f;
  constexpr float e_lo = (float)(1e-7 - (double)1e-7f);
  const float s = c + e_hi;
  const float bb = s - c;
  const float err = (c - (s - bb)) + (e_hi - bb);  // c + e_hi == s + err exactly
  const float dl0 = err + e_lo;
  const float dh = s + dl0;
  const float dl = dl0 - (dh - s);
  const float q0 = __fdiv_rn(b, dh);
  float r = __fmaf_rn(-q0, dh, b);
  r = __fmaf_rn(-q0, dl, r);
  return q0 + __fdiv_rn(r, dh);
}

// InitZ<true> (src/hfbs.cu:337-353): z = blur(b) / (blur(c) + 1e-7), the
// division in double as the reference's double literal makes it; h = 0.
__global__ void k_init_z(const float* __restrict__ blur_b, const float* __restrict__ blur_c,
                         float* __restrict__ z, float* __restrict__ h, long long n,
                         float* __restrict__ copy0, float* __restrict__ copy1) {
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < n;
       g += (long long)gridDim.x * blockDim.x) {
    const float v = div_by_c_plus_eps(blur_b[g], blur_c[g]);
    z[g] = v;
    h[g] = 0.f;
    if (copy0) copy0[g] = v;
    if (copy1) copy1[g] = v;
  }
}

// a16: SolveHFBS heavy-ball step (src/hfbs.cu:201-239).
__global__ void k_solve(const HInst* __restrict__ insts,
                        const float* __restrict__ zs, float* __restrict__ zd,
                        float* __restrict__ h, const float* __restrict__ norm,
                        const float* __restrict__ b,
                        const float* __restrict__ invA, float lambda,
                        float alpha, float beta) {
  const HInst I = insts[blockIdx.y];
  const int gx = I.gx, gy = I.gy, gl = I.gl;
  const float* z = zs + I.grid_off;
  const float* nn = norm + I.grid_off;
  const float* bb = b + I.grid_off;
  const float* ia = invA + I.grid_off;
  float* hh = h + I.grid_off;
  float* zo = zd + I.grid_off;
  const int sy = I.px, sz = I.px * gy;
  // one warp per grid row (fixed y, l); lanes stride along x
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < gy * gl;
       row += nwarps) {
    const int zz = row / gy, y = row - zz * gy;
    const int base = row * sy;
    // two x positions per lane per pass: their 34 loads are issued before
    // either result is computed
    for (int x0 = lane; x0 < gx; x0 += 64) {
      float d[2], zc[2], nc[2], bc[2], ic[2], hc[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int x = x0 + 32 * j;
        d[j] = zc[j] = nc[j] = bc[j] = ic[j] = hc[j] = 0.f;
        if (x < gx) {
          const int i = base + x;
          float a = 0.f;
          if (x > 0) a += z[i - 1] * nn[i - 1];
          if (x + 1 < gx) a += z[i + 1] * nn[i + 1];
          if (y > 0) a += z[i - sy] * nn[i - sy];
          if (y + 1 < gy) a += z[i + sy] * nn[i + sy];
          if (zz > 0) a += z[i - sz] * nn[i - sz];
          if (zz + 1 < gl) a += z[i + sz] * nn[i + sz];
          d[j] = a;
          zc[j] = z[i];
          nc[j] = nn[i];
          bc[j] = bb[i];
          ic[j] = ia[i];
          hc[j] = hh[i];
        }
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int x = x0 + 32 * j;
        if (x >= gx) break;
        const int i = base + x;
        const float q = (bc[j] + lambda * nc[j] * d[j]) * ic[j];
        const float grad = zc[j] - q;
        // |grad| > 1.345 with the double threshold of the reference: the
        // smallest float above 1.345 (double) is 1.345f
        const float gc = fabsf(grad) >= 1.345f ? copysignf(1.f, grad) : grad;
        const float hn = __fmaf_rn(beta, hc[j], gc);
        hh[i] = hn;
        zo[i] = zc[j] - alpha * hn;
      }
    }
  }
}

constexpr int kSliceXTable = 2048;

// The slice's corner values, once per solve: (count * z, count) at every
// voxel of (gx + 1) x (gy + 1) x (gl + 2), the overflow counts (times a zero
// z, as the reference's read past the grid gives) in plane gl and zeros on
// the faces past the grid, so that the slice reads its eight corners without
// tests.  count * z is the product the reference forms first.  One warp per
// (y, l) row of the padded grid.
__global__ void k_slice_pack(const HInst* __restrict__ insts, const float* __restrict__ count,
                             const float* __restrict__ ovf, const float* __restrict__ z,
                             float2* __restrict__ sgrid) {
  const HInst I = insts[blockIdx.y];
  const int PX = I.gx + 1, PY = I.gy + 1, rows = PY * (I.gl + 2);
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < rows; row += nwarps) {
    const int iz = row / PY, iy = row - iz * PY;
    float2* out = sgrid + I.slice_off + (long long)row * PX;
    for (int ix = lane; ix < PX; ix += 32) {
      float2 v = make_float2(0.f, 0.f);
      if (ix < I.gx && iy < I.gy) {
        if (iz < I.gl) {
          const long long g = gidx(I, ix, iy, iz);
          const float c = count[g];
          v = make_float2(c * z[g], c);
        } else if (iz == I.gl) {
          const float c = ovf[I.plane_off + (long long)iy * I.gx + ix];
          v = make_float2(c * 0.f, c);
        }
      }
      out[ix] = v;
    }
  }
}

__device__ __forceinline__ float slice_pixel(const HInst& I, const float2* __restrict__ sgrid,
                                             const HParams& p, int x, float fy, float fz,
                                             const float* fxt) {
  // x * 1.0f / sigma_x from the block's table where it covers x
  const float fx = x < kSliceXTable ? fxt[x] : (float)x * 1.0f / p.sigma_x;
  const float x0 = floorf(fx), y0 = floorf(fy), z0 = floorf(fz);
  const float wx = fx - x0, wy = fy - y0, wz = fz - z0;
  // x < W puts floor(x / sx) below gx (and likewise y, and L <= 255 puts
  // floor(L / sl) at most gl); the clamps only keep the reads inside the
  // padded grid
  const int ix = min((int)x0, I.gx - 1), iy = min((int)y0, I.gy - 1),
            iz = min((int)z0, I.gl);
  const int PX = I.gx + 1, PXY = PX * (I.gy + 1);
  const float2* c0 = sgrid + I.slice_off + (long long)iz * PXY + iy * PX + ix;
  float2 v[2][2][2];  // the eight corners' loads, all issued before the weighting
#pragma unroll
  for (int dz = 0; dz < 2; ++dz)
#pragma unroll
    for (int dy = 0; dy < 2; ++dy)
#pragma unroll
      for (int dx = 0; dx < 2; ++dx) v[dz][dy][dx] = c0[dz * PXY + dy * PX + dx];
  float num[2][2], den[2][2];
#pragma unroll
  for (int dz = 0; dz < 2; ++dz)
#pragma unroll
    for (int dy = 0; dy < 2; ++dy) {
      float ns = 0.f, ds = 0.f;
#pragma unroll
      for (int dx = 0; dx < 2; ++dx) {
        const float w = dx ? wx : 1.f - wx;
        ns += v[dz][dy][dx].x * w;
        ds += v[dz][dy][dx].y * w;
      }
      num[dz][dy] = ns;
      den[dz][dy] = ds;
    }
  const float c0y = num[0][0] * (1.f - wy) + num[0][1] * wy;
  const float c1y = num[1][0] * (1.f - wy) + num[1][1] * wy;
  const float c0m = den[0][0] * (1.f - wy) + den[0][1] * wy;
  const float c1m = den[1][0] * (1.f - wy) + den[1][1] * wy;
  return __fdiv_rn(c0y * (1.f - wz) + c1y * wz, c0m * (1.f - wz) + c1m * wz);
}

// a17: SliceSolution<true> (src/hfbs.cu:246-330): count-weighted trilinear
// interpolation of z at (x/sx, y/sy, L/sl).  One warp per image row, lanes
// along x, two pixels per lane per pass.
__global__ void k_slice(const HInst* __restrict__ insts,
                        const uchar4* __restrict__ guide,
                        const float2* __restrict__ sgrid, float* __restrict__ out,
                        HParams p) {
  // the reference's x/sx and L/sl (correctly rounded divisions) are the same
  // for every row: computed once per block into tables
  __shared__ float fxt[kSliceXTable];
  __shared__ float fzt[256];
  const HInst I = insts[blockIdx.y];
  for (int i = threadIdx.x; i < min(I.w, kSliceXTable); i += blockDim.x)
    fxt[i] = (float)i * 1.0f / p.sigma_x;
  for (int i = threadIdx.x; i < 256; i += blockDim.x) fzt[i] = (float)i * 1.0f / p.sigma_l;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  const uchar4* g = guide + I.pix_off;
  float* o = out + I.pix_off;
  for (int y = blockIdx.x * wpb + (threadIdx.x >> 5); y < I.h; y += gridDim.x * wpb) {
    const int row = y * I.pitch;
    const float fy = (float)y * 1.0f / p.sigma_y;
    // four pixels per lane per pass: their 32 corner loads are in flight
    // together
    for (int xb = lane; xb < I.w; xb += 128) {
      float zq[4], rq[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int x = xb + 32 * u;
        zq[u] = x < I.w ? fzt[g[row + x].x] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int x = min(xb + 32 * u, I.w - 1);  // past the width: a copy of the last
        rq[u] = slice_pixel(I, sgrid, p, x, fy, zq[u], fxt);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (xb + 32 * u < I.w) o[row + xb + 32 * u] = rq[u];
    }
  }
}

int blocks_for(long long n) {
  long long b = (n + kT - 1) / kT;
  if (b > 152 * 8) b = 152 * 8;
  return b < 1 ? 1 : (int)b;
}

}  // namespace

void hfbs_prepare_tma(const HfbsBatch& B, const HParams& p, cudaStream_t s) {
  if (!hfbs_uses_march(B)) return;
  std::vector<const float*> planes = {B.b, B.invA, B.z0, B.z1, B.h, B.t2, B.n0, B.n1, B.count};
  if (B.grad && B.grad->segment == 1)  // the kept iterates that start a march
    for (int it = 0; it < p.optim_iter_max; it += kHfbsMarchSteps)
      planes.push_back(B.grad->hist + (size_t)it * B.total_voxels);
  hfbs_march_prepare(B, planes, s);
}

bool hfbs_uses_march(const HfbsBatch& B) {
  return B.max_gl <= kHfbsMarchMaxGL && B.h_inst && B.solve_steps != 1;
}

int hfbs_launch_steps(const HfbsBatch& B, const HParams& p, const float* norm,
                      const float* zs, float* zd, const float* hs, float* hd, int steps,
                      float* rec, int rec_steps, cudaStream_t s) {
  ProfScope ps(s, DTSGB_K_HFBS_SOLVE);
  if (hfbs_uses_march(B))
    return hfbs_march_solve(B, hfbs_march_plan(B, 0, B.n_inst), p, norm, zs, zd, hs, hd, steps,
                            rec, rec_steps, s);
  // one step; h in place (hs == hd)
  const dim3 gr((unsigned)std::min<long long>((B.max_rows + 7) / 8, 4096), B.n_inst);
  k_solve<<<gr, kT, 0, s>>>(B.d_inst, zs, zd, hd, norm, B.b, B.invA, p.lambda, p.alpha, p.beta);
  DTSGB_CUDA(cudaGetLastError());
  return DTSGB_OK;
}

// The Laplace blur X -> Y -> Z of the pair (s0, s1) by way of (x0, x1) and (y0,
// y1) into (x0, x1); a field of the pair on each z of the grids (both in one
// thread took 10 us a sweep of 80 x 60 x 16, which waits on its loads; 8.6 along y
// and 2.8 along l so).
void hfbs_launch_blur_pair(const HfbsBatch& B, const HParams& p, const float* s0,
                           const float* s1, float* x0, float* x1, float* y0, float* y1,
                           cudaStream_t s) {
  const int ni = B.n_inst;
  // (rows: both fields in one warp where there are rows enough, whose warps
  // share their powers of beta: 64 ragged grids 125 us, 151 split)
  const dim3 gr((unsigned)std::min<long long>((B.max_rows + 7) / 8, 4096), ni,
                B.max_rows * ni > 152 * 64 ? 1 : 2);
  const dim3 gl_lines(blocks_for(B.max_lines), ni, 2);
  k_laplace_x<<<gr, kT, 0, s>>>(B.d_inst, s0, x0, s1, x1, p.neg_exp_beta);
  k_laplace<<<gl_lines, kT, 0, s>>>(B.d_inst, 1, x0, y0, x1, y1, p.neg_exp_beta);
  const dim3 gz((unsigned)std::min<long long>((B.max_cells + 127) / 128 + 1, 4096), ni, 2);
  if (B.max_gl <= 16)
    k_laplace_l<16><<<gz, 128, 0, s>>>(B.d_inst, y0, x0, y1, x1, p.neg_exp_beta);
  else if (B.max_gl <= 32)
    k_laplace_l<32><<<gz, 128, 0, s>>>(B.d_inst, y0, x0, y1, x1, p.neg_exp_beta);
  else
    k_laplace<<<gl_lines, kT, 0, s>>>(B.d_inst, 2, y0, x0, y1, x1, p.neg_exp_beta);
}

int hfbs_enqueue_solve(const HfbsBatch& B, const HParams& p, cudaStream_t s,
                       const float** z_final) {
  const int ni = B.n_inst;
  // row kernels: one warp per grid row, 8 warps per block
  const dim3 gr((unsigned)std::min<long long>((B.max_rows + 7) / 8, 4096), ni);
  // slice: one warp per image row, 8 rows per block
  long long max_h = 1;
  for (int i = 0; B.h_inst && i < ni; ++i) max_h = std::max<long long>(max_h, B.h_inst[i].h);
  if (!B.h_inst) max_h = (B.max_pixels + 31) / 32;
  const dim3 gp((unsigned)std::min<long long>((max_h + 7) / 8, 4096), ni);
  const dim3 gc((B.max_cells + 63) / 64, ni);
  const size_t splat_smem = sizeof(float) * 3 * (size_t)B.max_gl * 64;
  const size_t lbin_smem = sizeof(int) * 256;  // k_splat's luma table
  // a CTA per cell for large ones (k_splat_cell holds a bin per thread)
  const bool by_cell = (double)p.sigma_x * (double)p.sigma_y >= kSplatCellPx &&
                       B.max_gl < kSplatCellT;
  const dim3 gcell((unsigned)B.max_cells, ni);
  prof_begin(s, DTSGB_K_HFBS_SPLAT);
  if (by_cell && B.st == Storage::F32) {
    k_splat_cell<float><<<gcell, kSplatCellT, 0, s>>>(
        B.d_inst, B.guide, (const float*)B.target, (const float*)B.conf, B.count, B.csum, B.b,
        B.ovf, p);
  } else if (by_cell) {
    k_splat_cell<__nv_bfloat16><<<gcell, kSplatCellT, 0, s>>>(
        B.d_inst, B.guide, (const __nv_bfloat16*)B.target, (const __nv_bfloat16*)B.conf,
        B.count, B.csum, B.b, B.ovf, p);
  } else if (B.st == Storage::F32) {
    DTSGB_CUDA(allow_smem(k_splat<float>, splat_smem, lbin_smem));
    k_splat<float><<<gc, 64, splat_smem, s>>>(
        B.d_inst, B.guide, (const float*)B.target, (const float*)B.conf, B.count,
        B.csum, B.b, B.ovf, p);
  } else {
    DTSGB_CUDA(allow_smem(k_splat<__nv_bfloat16>, splat_smem, lbin_smem));
    k_splat<__nv_bfloat16><<<gc, 64, splat_smem, s>>>(
        B.d_inst, B.guide, (const __nv_bfloat16*)B.target,
        (const __nv_bfloat16*)B.conf, B.count, B.csum, B.b, B.ovf, p);
  }
  DTSGB_CUDA(cudaGetLastError());
  prof_end(s, DTSGB_K_HFBS_SPLAT);
  // bistochastization ping-pong: even iterations read the buffer filled with
  // ones, whose covered pad faces hold 1
  const int gflat = blocks_for(B.total_voxels);
  if (!B.reuse_norm) k_fill_ones<<<gflat, kT, 0, s>>>(B.n0, B.total_voxels);
  // The iterative stages (bistochastization, heavy-ball) touch only their own
  // instance's grid, so they run group by group: all iterations of a group
  // of consecutive instances whose grids fit in L2 before the next group,
  // which then streams from L2 instead of HBM after its first iteration.
  struct Group {
    int first, count;
    long long cols;  // max over the group of gx * gy
  };
  std::vector<Group> groups;
  if (B.h_inst && B.group_voxels > 0 && !B.grad) {
    Group g{0, 0, 0};
    long long vox = 0;
    for (int i = 0; i < ni; ++i) {
      const HInst& H = B.h_inst[i];
      const long long v = (long long)H.gx * H.gy * H.gl;
      if (g.count > 0 && vox + v > B.group_voxels) {
        groups.push_back(g);
        g = Group{i, 0, 0};
        vox = 0;
      }
      ++g.count;
      vox += v;
      g.cols = std::max(g.cols, (long long)H.gx * H.gy);
    }
    groups.push_back(g);
  } else {
    groups.push_back(Group{0, ni, B.max_cells});
  }
  // column kernels (bistochastization): one thread per (x, y)
  auto col_grid = [](const Group& g) {
    return dim3((unsigned)std::min<long long>((g.cols + kT - 1) / kT, 4096), g.count);
  };
  float* src = B.n0;
  float* dst = B.n1;
  for (const Group& g : groups) {
    src = B.n0;
    dst = B.n1;
    if (B.reuse_norm) {
      if (p.bistoch_iter_max % 2) std::swap(src, dst);
      continue;
    }
    const HfbsClusterPlan CP = hfbs_cluster_plan(B, g.first, g.count);
    if (CP.size > 0) {  // into the buffer the one-step ping-pong leaves it in
      if (p.bistoch_iter_max % 2) std::swap(src, dst);
      ProfScope ps(s, DTSGB_K_HFBS_BISTOCH);
      if (int st = hfbs_cluster_bistoch(B, CP, src, p.bistoch_iter_max, s)) return st;
    } else if (hfbs_uses_march(B)) {
      // up to kHfbsMarchSteps iterations per pass; one pass split in two when
      // the number of passes and of iterations differ in parity, so that the
      // result lands in the buffer the one-step ping-pong leaves it in
      constexpr int K = kHfbsMarchSteps;
      std::vector<int> plan;
      for (int r = p.bistoch_iter_max; r > 0; r -= K) plan.push_back(std::min(K, r));
      if ((int)(plan.size() % 2) != p.bistoch_iter_max % 2) {
        for (int i = (int)plan.size() - 1; i >= 0; --i)
          if (plan[i] >= 2) {
            const int a = plan[i] / 2;
            plan[i] -= a;
            plan.insert(plan.begin() + i + 1, a);
            break;
          }
      }
      const HfbsMarchPlan P = hfbs_march_plan(B, g.first, g.count);
      int it0 = 0;
      for (int steps : plan) {
        ProfScope ps(s, DTSGB_K_HFBS_BISTOCH);
        if (int st = hfbs_march_bistoch(B, P, src, dst, it0, steps, s)) return st;
        std::swap(src, dst);
        it0 += steps;
      }
    } else {
      for (int it = 0; it < p.bistoch_iter_max; ++it) {
        prof_begin(s, DTSGB_K_HFBS_BISTOCH);
        DTSGB_CUDA(launch_dependent(k_bistoch, col_grid(g), dim3(kT), 0, s, B.d_inst + g.first,
                                    src, dst, B.count, (it % 2 == 0) ? 1.f : 0.f));
        prof_end(s, DTSGB_K_HFBS_BISTOCH);
        std::swap(src, dst);
      }
    }
  }
  float* norm = src;
  float* spare = dst;
  prof_begin(s, DTSGB_K_HFBS_OTHER);
  k_inv_diag<<<gflat, kT, 0, s>>>(B.count, B.csum, norm, B.invA, p.lambda,
                                  B.total_voxels);
  // Laplace blur of (c, b)
  hfbs_launch_blur_pair(B, p, B.csum, B.b, B.t0, B.t1, B.t2, spare, s);
  // blur_c = t0, blur_b = t1
  // z_0 is overwritten: kept for inspection, and as the adjoint's first iterate
  float* z_kept = B.grad && B.grad->segment == 1 && p.optim_iter_max > 0 ? B.grad->hist : nullptr;
  k_init_z<<<gflat, kT, 0, s>>>(B.t1, B.t0, B.z0, B.h, B.total_voxels,
                                B.keep_debug ? B.dbg_z_init : nullptr, z_kept);
  prof_end(s, DTSGB_K_HFBS_OTHER);
  float* zs = B.z0;
  float* zd = B.z1;
  if (B.grad) {
    // iterates kept for the adjoint (HfbsGradState)
    const HfbsGradState& G = *B.grad;
    const int K = p.optim_iter_max, S = G.segment;
    const bool tb = hfbs_uses_march(B);
    const long long tv = B.total_voxels;
    const size_t gbytes = (size_t)tv * sizeof(float);
    const HfbsClusterPlan CP = hfbs_cluster_plan(B, 0, ni);
    if (S == 1 && CP.size > 0 && K > 0) {
      ProfScope ps(s, DTSGB_K_HFBS_SOLVE);
      if (int st = hfbs_cluster_solve(B, CP, p, norm, B.z0, B.z1, B.h, nullptr, K, G.hist + tv,
                                      K - 1, s))
        return st;
      zs = B.z1;
    } else if (S == 1) {
      // z_k in hist plane k; h ping-pongs through the free blur temporary t2
      float* hs = B.h;
      float* hd = tb ? B.t2 : B.h;
      for (int it = 0; it < K;) {
        const int steps = tb ? std::min(kHfbsMarchSteps, K - it) : 1;
        float* zout = it + steps < K ? G.hist + (size_t)(it + steps) * tv : B.z1;
        const int rec_steps = tb ? std::min(steps, K - 1 - it) : 0;
        if (int st = hfbs_launch_steps(B, p, norm, G.hist + (size_t)it * tv, zout, hs, hd, steps,
                                       G.hist + (size_t)(it + 1) * tv, rec_steps, s))
          return st;
        std::swap(hs, hd);
        it += steps;
      }
      zs = K > 0 ? B.z1 : B.z0;
    } else {
      // z and h at the start of every segment
      float* hs = B.h;
      float* hd = tb ? B.t2 : B.h;
      for (int it = 0; it < K;) {
        if (it % S == 0) {
          DTSGB_CUDA(cudaMemcpyAsync(G.ckz + (size_t)(it / S) * tv, zs, gbytes,
                                     cudaMemcpyDeviceToDevice, s));
          DTSGB_CUDA(cudaMemcpyAsync(G.ckh + (size_t)(it / S) * tv, hs, gbytes,
                                     cudaMemcpyDeviceToDevice, s));
        }
        const int steps = tb ? std::min({kHfbsMarchSteps, K - it, S - it % S}) : 1;
        if (int st = hfbs_launch_steps(B, p, norm, zs, zd, hs, hd, steps, nullptr, 0, s))
          return st;
        std::swap(zs, zd);
        std::swap(hs, hd);
        it += steps;
      }
    }
  } else if (hfbs_uses_march(B)) {
    // h ping-pongs through the free blur temporary t2 (its final value is not
    // needed)
    for (const Group& g : groups) {
      zs = B.z0;
      zd = B.z1;
      float* hs = B.h;
      float* hd = B.t2;
      const HfbsClusterPlan CP = hfbs_cluster_plan(B, g.first, g.count);
      if (CP.size > 0 && p.optim_iter_max > 0) {
        // (every group ends in the buffer its marches would leave it in)
        if ((p.optim_iter_max + kHfbsMarchSteps - 1) / kHfbsMarchSteps % 2 == 0) zd = B.z0;
        ProfScope ps(s, DTSGB_K_HFBS_SOLVE);
        if (int st = hfbs_cluster_solve(B, CP, p, norm, zs, zd, hs, nullptr, p.optim_iter_max,
                                        nullptr, 0, s))
          return st;
        zs = zd;
        continue;
      }
      const HfbsMarchPlan P = hfbs_march_plan(B, g.first, g.count);
      for (int it = 0; it < p.optim_iter_max; it += kHfbsMarchSteps) {
        const int steps = std::min(kHfbsMarchSteps, p.optim_iter_max - it);
        ProfScope ps(s, DTSGB_K_HFBS_SOLVE);
        if (int st = hfbs_march_solve(B, P, p, norm, zs, zd, hs, hd, steps, nullptr, 0, s))
          return st;
        std::swap(zs, zd);
        std::swap(hs, hd);
      }
    }
  } else
  for (const Group& g : groups) {
    zs = B.z0;
    zd = B.z1;
    long long rows = 0;  // one warp per grid row (y, l) of the group's largest grid
    for (int i = 0; i < g.count; ++i)
      rows = B.h_inst ? std::max(rows, (long long)B.h_inst[g.first + i].gy *
                                           B.h_inst[g.first + i].gl)
                      : B.max_rows;
    const dim3 gr_g((unsigned)std::min<long long>((rows + 7) / 8, 4096), g.count);
    for (int it = 0; it < p.optim_iter_max; ++it) {
      prof_begin(s, DTSGB_K_HFBS_SOLVE);
      k_solve<<<gr_g, kT, 0, s>>>(B.d_inst + g.first, zs, zd, B.h, norm, B.b, B.invA,
                                  p.lambda, p.alpha, p.beta);
      prof_end(s, DTSGB_K_HFBS_SOLVE);
      std::swap(zs, zd);
    }
  }
  if (z_final) *z_final = zs;
  prof_begin(s, DTSGB_K_HFBS_SLICE);
  long long prows = 1;  // rows of the largest padded slice grid
  for (int i = 0; B.h_inst && i < ni; ++i)
    prows = std::max<long long>(prows, (long long)(B.h_inst[i].gy + 1) * (B.h_inst[i].gl + 2));
  if (!B.h_inst) prows = B.max_lines + 2 * B.max_rows + 260;
  const dim3 gsl((unsigned)std::min<long long>((prows + 7) / 8, 4096), ni);
  k_slice_pack<<<gsl, kT, 0, s>>>(B.d_inst, B.count, B.ovf, zs, B.sgrid);
  k_slice<<<gp, kT, 0, s>>>(B.d_inst, B.guide, B.sgrid, B.out, p);
  prof_end(s, DTSGB_K_HFBS_SLICE);
  DTSGB_CUDA(cudaGetLastError());
  return DTSGB_OK;
}

}  // namespace dtsgb
