// The iterative HFBS stages on grids small enough to stay on chip: all
// heavy-ball steps (src/hfbs.cu:201-239), or all bistochastization iterations
// (src/hfbs.cu:126-155), of an instance in one launch of one thread-block
// cluster.
//
// Each CTA of the cluster owns a slab of grid rows y; a thread owns items of
// four levels of one (x, y) column and keeps their z, h, n, b and invA in
// registers for the whole solve.  Per step the products z * n go to shared
// memory (two buffers in turn, the four levels of an item side by side: one
// 16-byte access), those of a slab's first and last row also to
// the neighbouring CTA's halo row through distributed shared memory; one
// cluster barrier later every neighbour is a local read.  Memory is touched
// before the first and after the last step only.
//
// Bound by latency: a step is one exchange (6 shared-memory reads per four
// voxels) and one cluster barrier.  Measured: 140 steps on a 22 x 17 x 16 grid
// in 71 us, 64 on 80 x 60 x 16 in 109 with every iterate recorded (89 and 117
// with planes of levels, 18 reads per four voxels); a launch per four steps, the
// form this replaces, took 12 to 16 us on such grids whatever their size (a
// launch, a round of loads and four block barriers).
//
// Taken where every instance of the launch fits: per CTA 2048 items (8192
// voxels; registers) and 227 KB of the two buffers, so 131072 voxels for 16
// CTAs.  On such grids it beats the march (hfbs_march.cu) also when many run
// side by side, since nothing is recomputed at block borders.
//
// Out-of-grid values, neighbour order and arithmetic are the march's
// (hfbs_march.cu): the results are the same bit for bit.
#include <algorithm>
#include <vector>

#include "../../include/dtsgb.h"
#include "dtsgb_internal.cuh"
#include "hfbs_internal.cuh"

namespace dtsgb {
namespace {

constexpr int kCV = 4;  // levels of an item
// Threads a CTA may have when each owns that many items (registers: 20 an
// item and about 45), and items a CTA can hold.
__host__ __device__ constexpr int max_threads(int ipt) {
  return ipt == 1 ? 1024 : ipt == 2 ? 768 : ipt == 3 ? 576 : 512;
}
// The same of the adjoint (44 registers an item).
__host__ __device__ constexpr int adj_threads(int ipt) { return ipt == 1 ? 704 : 640; }
constexpr int kAdjItems = 2;
constexpr int kCItems = 4;

struct ClusterArgs {
  const float *z, *h, *n, *b, *a;  // normalisation: n the counts
  float *zd, *hd;                  // hd null: h is not needed afterwards
  float* rec;                      // z after step k + 1 in plane k, rec_steps of them
  long long rec_stride;
  int rec_steps, steps;
  float lambda, alpha, beta;
};

enum { kHeavyBall = 0, kBistoch = 1 };

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned n;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
  return n;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;"
               ::: "memory");
}
// Stores v at the address that `local` has in the shared memory of CTA `rank`.
__device__ __forceinline__ void store_remote(const float4* local, unsigned rank, float4 v) {
  unsigned a = (unsigned)__cvta_generic_to_shared(local), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(r), "f"(v.x), "f"(v.y),
               "f"(v.z), "f"(v.w)
               : "memory");
}
// Level v of an item's four.
__device__ __forceinline__ float lev(const float4& q, int v) {
  return v == 0 ? q.x : v == 1 ? q.y : v == 2 ? q.z : q.w;
}

// Rows of a CTA's slab, items of a CTA and its shared memory for a cluster of
// `c` CTAs.
__host__ __device__ inline int slab_rows(int gy, int c) { return (gy + c - 1) / c; }
inline long long slab_items(const HInst& H, int c) {
  return (long long)slab_rows(H.gy, c) * H.gx * ((H.gl + kCV - 1) / kCV);
}
inline size_t slab_smem(const HInst& H, int c) {  // of one buffer
  return sizeof(float) * (size_t)((H.gl + kCV - 1) / kCV * kCV) *
         (slab_rows(H.gy, c) + 2) * (H.gx + 2);
}

template <int MODE, bool REC, int IPT>
__global__ void __launch_bounds__(max_threads(IPT), 1)
    k_hfbs_cluster(const HInst* __restrict__ insts, ClusterArgs A) {
  extern __shared__ float4 smc[];  // [buffer][group of levels][R + 2][gx + 2]
  const HInst I = insts[blockIdx.y];
  const int gx = I.gx, gy = I.gy, gl = I.gl;
  const int rank = (int)cluster_rank(), C = (int)cluster_size();
  const int R = slab_rows(gy, C), nlc = (gl + kCV - 1) / kCV;
  const int gxp = gx + 2, PS = (R + 2) * gxp, BUF = nlc * PS;
  const int tid = threadIdx.x, T = blockDim.x;
  for (int i = tid; i < 2 * BUF; i += T) smc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  if (MODE == kBistoch) {
    // the covered pad faces read 1 on even iterations (the first buffer), 0 on
    // odd ones
    const int rows = min(R, gy - rank * R);  // may be <= 0
    auto at = [&](int l, int r, int x) -> float& {
      return reinterpret_cast<float*>(smc + (l / kCV) * PS + r * gxp + x)[l % kCV];
    };
    if (I.cov_x)
      for (int i = tid; i < gl * max(rows, 0); i += T) {
        const int l = i / rows, yy = i - l * rows;
        at(l, yy + 1, gx + 1) = 1.f;
      }
    if (I.cov_y && rows > 0 && rank * R + rows == gy)
      for (int i = tid; i < gl * gx; i += T) {
        const int l = i / gx, x = i - l * gx;
        at(l, rows + 1, x + 1) = 1.f;
      }
  }
  const int items = R * gx * nlc, plane = I.px * gy;
  float z[IPT][kCV], h[IPT][kCV], n[IPT][kCV], b[IPT][kCV], a[IPT][kCV];
  int o[IPT];        // index of the item in a buffer
  int lc[IPT];       // its group of levels (-1: no item)
  int edge[IPT];     // bit 0: first row of the slab, bit 1: last
  long long g[IPT];  // element of level 0 in a grid plane
#pragma unroll
  for (int j = 0; j < IPT; ++j) {
    const int i = tid + j * T;
    lc[j] = -1;
    o[j] = edge[j] = 0;
    g[j] = 0;
#pragma unroll
    for (int v = 0; v < kCV; ++v) z[j][v] = h[j][v] = n[j][v] = b[j][v] = a[j][v] = 0.f;
    if (i < items) {
      const int c = i / (R * gx), q = i - c * (R * gx), yy = q / gx, x = q - yy * gx;
      const int y = rank * R + yy;
      if (y < gy) {
        lc[j] = c;
        o[j] = c * PS + (yy + 1) * gxp + x + 1;
        edge[j] = (yy == 0 && rank > 0 ? 1 : 0) | (yy == R - 1 && rank + 1 < C ? 2 : 0);
        g[j] = I.grid_off + (long long)c * kCV * plane + (long long)y * I.px + x;
#pragma unroll
        for (int v = 0; v < kCV; ++v)
          if (c * kCV + v < gl) {
            const long long gv = g[j] + (long long)v * plane;
            n[j][v] = A.n[gv];
            if (MODE == kHeavyBall) {
              z[j][v] = A.z[gv];
              h[j][v] = A.h[gv];
              b[j][v] = A.b[gv];
              a[j][v] = A.a[gv];
            } else {
              z[j][v] = 1.f;
            }
          }
      }
    }
  }
  // every CTA of the cluster runs and its buffers are zeroed
  cluster_barrier();
  for (int s = 0; s < A.steps; ++s) {
    float4* P = smc + (s & 1) * BUF;
    float p[IPT][kCV];
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
#pragma unroll
      for (int v = 0; v < kCV; ++v)
        p[j][v] = MODE == kHeavyBall ? __fmul_rn(z[j][v], n[j][v]) : z[j][v];
      if (lc[j] >= 0) {
        float4* q = P + o[j];
        const float4 p4 = make_float4(p[j][0], p[j][1], p[j][2], p[j][3]);
        *q = p4;
        if (edge[j] & 1) store_remote(q + R * gxp, rank - 1, p4);
        if (edge[j] & 2) store_remote(q - R * gxp, rank + 1, p4);
      }
    }
    cluster_barrier();
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
      if (lc[j] < 0) continue;
      const float4* q = P + o[j];
      const float lo = lc[j] > 0 ? q[-PS].w : 0.f;
      const float hi = lc[j] + 1 < nlc ? q[PS].x : 0.f;
      const float4 xm = q[-1], xp = q[1], ym = q[-gxp], yp = q[gxp];
      const float pz = MODE == kBistoch && I.cov_l && !(s & 1) ? 1.f : 0.f;
#pragma unroll
      for (int v = 0; v < kCV; ++v) {
        const float below = v > 0 ? p[j][v > 0 ? v - 1 : 0] : lo;
        float above = v + 1 < kCV ? p[j][v + 1 < kCV ? v + 1 : v] : hi;
        if (MODE == kHeavyBall) {
          hfbs_step(lev(xm, v), lev(xp, v), lev(ym, v), lev(yp, v), below, above, n[j][v],
                    b[j][v], a[j][v], A.lambda, A.alpha, A.beta, z[j][v], h[j][v]);
        } else if (lc[j] * kCV + v < gl) {
          if (lc[j] * kCV + v + 1 == gl) above = pz;
          float t = lev(xm, v);
          t += lev(xp, v);
          t += lev(ym, v);
          t += lev(yp, v);
          t += below;
          t += above;
          const float blurred = 2.f * p[j][v] + t;
          z[j][v] = __fsqrt_rn(__fdiv_rn(p[j][v] * (n[j][v] + 0.00001f), blurred + 0.00001f));
        }
      }
      if (REC && s < A.rec_steps) {
        float* r = A.rec + s * A.rec_stride + g[j];
#pragma unroll
        for (int v = 0; v < kCV; ++v)
          if (lc[j] * kCV + v < gl) r[(long long)v * plane] = z[j][v];
      }
    }
  }
#pragma unroll
  for (int j = 0; j < IPT; ++j) {
    if (lc[j] < 0) continue;
#pragma unroll
    for (int v = 0; v < kCV; ++v)
      if (lc[j] * kCV + v < gl) {
        const long long gv = g[j] + (long long)v * plane;
        A.zd[gv] = z[j][v];
        if (MODE == kHeavyBall && A.hd) A.hd[gv] = h[j][v];
      }
  }
}

// ---- the adjoint ---------------------------------------------------------------
struct ClusterAdjArgs {
  const float *hist, *n, *b, *a;
  float *gz, *gb, *ginv;
  long long stride;  // voxels of an iterate
  int steps;
  float lambda, alpha, beta;
};

// All steps of the heavy-ball adjoint, from the last: the same ownership and
// exchange as the solve, with two products per step to exchange (z_k * n of the
// forward iterate, and gw of the step after it, which completes gz) and the
// next iterate's loads in flight during a step.  64 steps on 80 x 60 x 16:
// 192 us (238 with planes of levels), 384 by a launch per step; bound by the
// shared memory's bandwidth (13 words a voxel-step) and the barrier of a step.
template <int IPT>
__global__ void __launch_bounds__(adj_threads(IPT), 1)
    k_hfbs_cluster_adj(const HInst* __restrict__ insts, ClusterAdjArgs A) {
  extern __shared__ float4 smc[];  // [buffer][group of levels][R + 2][gx + 2]
  const HInst I = insts[blockIdx.y];
  const int gx = I.gx, gy = I.gy, gl = I.gl;
  const int rank = (int)cluster_rank(), C = (int)cluster_size();
  const int R = slab_rows(gy, C), nlc = (gl + kCV - 1) / kCV;
  const int gxp = gx + 2, PS = (R + 2) * gxp, BUF = nlc * PS;
  const int tid = threadIdx.x, T = blockDim.x;
  for (int i = tid; i < 4 * BUF; i += T) smc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int items = R * gx * nlc, plane = I.px * gy;
  float z[IPT][kCV], n[IPT][kCV], b[IPT][kCV], a[IPT][kCV];
  float gz[IPT][kCV], gh[IPT][kCV], gb[IPT][kCV], gi[IPT][kCV], gg[IPT][kCV];
  int o[IPT], lc[IPT], edge[IPT], g[IPT];
  const float* zk = A.hist + I.grid_off + (long long)(A.steps - 1) * A.stride;
  A.n += I.grid_off;
  A.b += I.grid_off;
  A.a += I.grid_off;
  A.gz += I.grid_off;
  A.gb += I.grid_off;
  A.ginv += I.grid_off;
#pragma unroll
  for (int j = 0; j < IPT; ++j) {
    const int i = tid + j * T;
    lc[j] = -1;
    o[j] = edge[j] = 0;
    g[j] = 0;
#pragma unroll
    for (int v = 0; v < kCV; ++v)
      z[j][v] = n[j][v] = b[j][v] = a[j][v] = gz[j][v] = gh[j][v] = gb[j][v] = gi[j][v] =
          gg[j][v] = 0.f;
    if (i < items) {
      const int c = i / (R * gx), q = i - c * (R * gx), yy = q / gx, x = q - yy * gx;
      const int y = rank * R + yy;
      if (y < gy) {
        lc[j] = c;
        o[j] = c * PS + (yy + 1) * gxp + x + 1;
        edge[j] = (yy == 0 && rank > 0 ? 1 : 0) | (yy == R - 1 && rank + 1 < C ? 2 : 0);
        g[j] = c * kCV * plane + y * I.px + x;
#pragma unroll
        for (int v = 0; v < kCV; ++v)
          if (c * kCV + v < gl) {
            const int gv = g[j] + v * plane;
            z[j][v] = zk[gv];
            n[j][v] = A.n[gv];
            b[j][v] = A.b[gv];
            a[j][v] = A.a[gv];
            gz[j][v] = A.gz[gv];
          }
      }
    }
  }
  // every CTA of the cluster runs and its buffers are zeroed
  __syncthreads();
  cluster_barrier();
  for (int s = 0; s <= A.steps; ++s) {  // the last pass only completes gz
    float4* P = smc + (s & 1) * BUF;
    float4* G = smc + (2 + (s & 1)) * BUF;
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
      if (lc[j] < 0) continue;
      float p[kCV], w[kCV];
#pragma unroll
      for (int v = 0; v < kCV; ++v) {
        p[v] = __fmul_rn(z[j][v], n[j][v]);
        w[v] = hfbs_adj_product(n[j][v], a[j][v], gg[j][v]);
      }
      const float4 p4 = make_float4(p[0], p[1], p[2], p[3]);
      const float4 w4 = make_float4(w[0], w[1], w[2], w[3]);
      float4 *qp = P + o[j], *qg = G + o[j];
      *qp = p4;
      *qg = w4;
      if (edge[j] & 1) {
        store_remote(qp + R * gxp, rank - 1, p4);
        store_remote(qg + R * gxp, rank - 1, w4);
      }
      if (edge[j] & 2) {
        store_remote(qp - R * gxp, rank + 1, p4);
        store_remote(qg - R * gxp, rank + 1, w4);
      }
    }
    // the next iterate, in flight over the barrier and this step
    float zn[IPT][kCV];
    zk -= A.stride;
#pragma unroll
    for (int j = 0; j < IPT; ++j)
#pragma unroll
      for (int v = 0; v < kCV; ++v)
        zn[j][v] = s + 1 < A.steps && lc[j] >= 0 && lc[j] * kCV + v < gl
                       ? zk[g[j] + v * plane]
                       : 0.f;
    cluster_barrier();
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
      if (lc[j] < 0) continue;
      // the neighbour sums of four levels, in the order x, y, l
      auto sums = [&](const float4* q, float (&t)[kCV]) {
        const float4 xm = q[-1], xp = q[1], ym = q[-gxp], yp = q[gxp], c = q[0];
        const float lo = lc[j] > 0 ? q[-PS].w : 0.f;
        const float hi = lc[j] + 1 < nlc ? q[PS].x : 0.f;
#pragma unroll
        for (int v = 0; v < kCV; ++v) {
          t[v] = __fadd_rn(__fadd_rn(__fadd_rn(lev(xm, v), lev(xp, v)), lev(ym, v)), lev(yp, v));
          t[v] = __fadd_rn(t[v], v > 0 ? lev(c, v > 0 ? v - 1 : 0) : lo);
          t[v] = __fadd_rn(t[v], v + 1 < kCV ? lev(c, v + 1 < kCV ? v + 1 : v) : hi);
        }
      };
      float t[kCV];
      if (s > 0) {
        sums(G + o[j], t);
#pragma unroll
        for (int v = 0; v < kCV; ++v)
          gz[j][v] = hfbs_finish_adj(gz[j][v], gg[j][v], n[j][v], t[v], A.lambda);
      }
      if (s < A.steps) {
        sums(P + o[j], t);
#pragma unroll
        for (int v = 0; v < kCV; ++v)
          hfbs_step_adj(t[v], z[j][v], n[j][v], b[j][v], a[j][v], gz[j][v], A.lambda, A.alpha,
                        A.beta, gh[j][v], gb[j][v], gi[j][v], gg[j][v]);
      }
    }
#pragma unroll
    for (int j = 0; j < IPT; ++j)
#pragma unroll
      for (int v = 0; v < kCV; ++v) z[j][v] = zn[j][v];
  }
#pragma unroll
  for (int j = 0; j < IPT; ++j) {
    if (lc[j] < 0) continue;
#pragma unroll
    for (int v = 0; v < kCV; ++v)
      if (lc[j] * kCV + v < gl) {
        const int gv = g[j] + v * plane;
        A.gz[gv] = gz[j][v];
        A.gb[gv] = gb[j][v];
        A.ginv[gv] = gi[j][v];
      }
  }
}

// Launches a kernel with one cluster of P.size CTAs per instance, or (clusters
// given) only asks how many such clusters can be resident.
template <typename F, typename Args>
cudaError_t launch_cluster(F* kern, const HfbsBatch& B, const HfbsClusterPlan& P, const Args& A,
                           cudaStream_t s, int* clusters) {
  cudaError_t e = allow_smem(kern, P.smem);
  if (e == cudaSuccess && P.size > 8)
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = P.size;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(P.size, P.count);
  c.blockDim = dim3(P.threads);
  c.dynamicSmemBytes = P.smem;
  c.stream = s;
  c.attrs = at;
  c.numAttrs = 1;
  if (clusters) return cudaOccupancyMaxActiveClusters(clusters, kern, &c);
  return cudaLaunchKernelEx(&c, kern, B.d_inst + P.first, A);
}

template <int MODE, bool REC, int IPT>
cudaError_t launch(const HfbsBatch& B, const HfbsClusterPlan& P, const ClusterArgs& A,
                   cudaStream_t s, int* clusters) {
  return launch_cluster(k_hfbs_cluster<MODE, REC, IPT>, B, P, A, s, clusters);
}

template <int MODE, bool REC>
cudaError_t launch_items(const HfbsBatch& B, const HfbsClusterPlan& P, const ClusterArgs& A,
                         cudaStream_t s, int* clusters = nullptr) {
  switch (P.items) {
    case 1: return launch<MODE, REC, 1>(B, P, A, s, clusters);
    case 2: return launch<MODE, REC, 2>(B, P, A, s, clusters);
    case 3: return launch<MODE, REC, 3>(B, P, A, s, clusters);
  }
  return launch<MODE, REC, kCItems>(B, P, A, s, clusters);
}

cudaError_t launch_adj(const HfbsBatch& B, const HfbsClusterPlan& P, const ClusterAdjArgs& A,
                       cudaStream_t s, int* clusters = nullptr) {
  return P.items <= 1 ? launch_cluster(k_hfbs_cluster_adj<1>, B, P, A, s, clusters)
                      : launch_cluster(k_hfbs_cluster_adj<2>, B, P, A, s, clusters);
}

}  // namespace

// The cluster of up to 16 CTAs that holds every instance with up to most_items
// items a thread (threads(items) of them) and `buffers` exchange buffers; size 0
// where an instance does not fit.
template <typename T>
static HfbsClusterPlan plan_cluster(const HfbsBatch& B, int first, int count, int most_items,
                                    T threads, int buffers) {
  HfbsClusterPlan P;
  if (!hfbs_uses_march(B)) return P;
  int min_gy = 1 << 30;
  for (int i = 0; i < count; ++i) min_gy = std::min(min_gy, B.h_inst[first + i].gy);
  for (int c = 16; c >= 1; c /= 2) {
    if (c > 1 && c > min_gy) continue;
    long long items = 0;
    size_t smem = 0;
    for (int i = 0; i < count; ++i) {
      items = std::max(items, slab_items(B.h_inst[first + i], c));
      smem = std::max(smem, buffers * slab_smem(B.h_inst[first + i], c));
    }
    if (items > (long long)most_items * threads(most_items) || smem > kMaxSmem)
      break;  // smaller clusters hold less
    P.size = c;
    P.items = 1;
    while (items > (long long)P.items * threads(P.items)) ++P.items;
    P.threads = (int)((items + P.items - 1) / P.items + 31) / 32 * 32;
    P.smem = smem;
    P.first = first;
    P.count = count;
    // the largest cluster whose instances run side by side
    if ((long long)c * count <= 128) break;
  }
  return P;
}

HfbsClusterPlan hfbs_cluster_plan(const HfbsBatch& B, int first, int count) {
  HfbsClusterPlan P = plan_cluster(B, first, count, kCItems, max_threads, 2);
  int n = 0;
  if (P.size > 0 &&
      (launch_items<kHeavyBall, false>(B, P, ClusterArgs{}, nullptr, &n) != cudaSuccess || n < 1)) {
    (void)cudaGetLastError();
    P.size = 0;
  }
  return P;
}

HfbsClusterPlan hfbs_cluster_adj_plan(const HfbsBatch& B) {
  HfbsClusterPlan P = plan_cluster(B, 0, B.n_inst, kAdjItems, adj_threads, 4);
  int n = 0;
  if (P.size > 0 && (launch_adj(B, P, ClusterAdjArgs{}, nullptr, &n) != cudaSuccess || n < 1)) {
    (void)cudaGetLastError();
    P.size = 0;
  }
  return P;
}

int hfbs_cluster_adjoint(const HfbsBatch& B, const HfbsClusterPlan& P, const HParams& p,
                         const float* norm, const float* hist, float* gz, float* gb, float* ginv,
                         int steps, cudaStream_t s) {
  const ClusterAdjArgs A{hist, norm, B.b, B.invA, gz, gb, ginv, B.total_voxels, steps,
                         p.lambda, p.alpha, p.beta};
  DTSGB_CUDA(launch_adj(B, P, A, s));
  return DTSGB_OK;
}

int hfbs_cluster_solve(const HfbsBatch& B, const HfbsClusterPlan& P, const HParams& p,
                       const float* norm, const float* zs, float* zd, const float* hs, float* hd,
                       int steps, float* rec, int rec_steps, cudaStream_t s) {
  const ClusterArgs A{zs, hs, norm, B.b, B.invA, zd, hd, rec, B.total_voxels, rec_steps, steps,
                      p.lambda, p.alpha, p.beta};
  if (rec_steps > 0) DTSGB_CUDA((launch_items<kHeavyBall, true>(B, P, A, s)));
  else DTSGB_CUDA((launch_items<kHeavyBall, false>(B, P, A, s)));
  return DTSGB_OK;
}

int hfbs_cluster_bistoch(const HfbsBatch& B, const HfbsClusterPlan& P, float* dst, int steps,
                         cudaStream_t s) {
  const ClusterArgs A{nullptr, nullptr, B.count, nullptr, nullptr, dst, nullptr, nullptr, 0, 0,
                      steps, 0.f, 0.f, 0.f};
  DTSGB_CUDA((launch_items<kBistoch, false>(B, P, A, s)));
  return DTSGB_OK;
}

}  // namespace dtsgb
