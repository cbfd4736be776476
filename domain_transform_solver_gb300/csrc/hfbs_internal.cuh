// Internal HFBS declarations (not part of the C ABI).
#pragma once

#include "dtsgb_internal.cuh"
#include "tma.cuh"

namespace dtsgb {

// One HFBS instance: its image plane (shared layout with the DTS planes)
// and its bilateral grid.
struct HInst {
  int w, h, pitch;
  int gx, gy, gl;
  // row pitch of the grids in voxels: gx rounded up to a multiple of 4, so
  // that every grid row starts on a 16-byte boundary (tensor-map tiles);
  // voxel (x, y, l) is at grid_off + (l * gy + y) * px + x, and the voxels
  // x >= gx of a row are padding that no stencil reads
  int px;
  // pad faces written by the reference's FillGrid (g % 8 != 0 and inside
  // the max-size allocation); they read the last fill value of the buffer
  int cov_x, cov_y, cov_l;
  // luma bin == gl is stored (and read back by the slice) only when the
  // z = gl plane lies inside the allocation
  int ovf_stored;
  long long pix_off;    // element offset of pixel (0,0)
  long long grid_off;   // element offset of voxel (0,0,0)
  long long plane_off;  // element offset of the overflow count plane
  // float2 offset of the slice grid: (count * z, count) over (gx + 1) x
  // (gy + 1) x (gl + 2) voxels, zero past the grid and the overflow counts
  // in plane gl (see k_slice_pack)
  long long slice_off;
};

// First pixel index p >= 0 with floorf(p * 1.0f / sigma) >= cell (the
// reference's bin of pixel p, src/hfbs.cu:82-83); n if none.
__device__ __forceinline__ int cell_start(int cell, float sigma, int n) {
  int p = (int)ceilf((float)cell * sigma) - 2;
  if (p < 0) p = 0;
  if (p > n) p = n;
  while (p < n && (int)floorf((float)p * 1.0f / sigma) < cell) ++p;
  while (p > 0 && (int)floorf((float)(p - 1) * 1.0f / sigma) >= cell) --p;
  return p;
}

// One heavy-ball step of one voxel (src/hfbs.cu:201-239): the rounded products
// z * n of its neighbours in the reference's order, n, b, invA, and z and h
// updated in place.  Every operation is spelled out, so that all kernels that
// step give the same bits.
__device__ __forceinline__ void hfbs_step(float xm, float xp, float ym, float yp, float lm,
                                          float lp, float n, float b, float a, float lambda,
                                          float alpha, float beta, float& z, float& h) {
  const float d = __fadd_rn(
      __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(xm, xp), ym), yp), lm), lp);
  const float t = __fmaf_rn(__fmul_rn(lambda, n), d, b);
  const float grad = __fmaf_rn(-t, a, z);
  // |grad| > 1.345 with the double threshold of the reference: the smallest
  // float above 1.345 (double) is 1.345f
  const float gc = fabsf(grad) >= 1.345f ? copysignf(1.f, grad) : grad;
  h = __fmaf_rn(beta, h, gc);
  z = __fmaf_rn(-alpha, h, z);
}

// The adjoint of a heavy-ball step of one voxel, in two parts that lie one
// exchange apart.  hfbs_step_adj: from the neighbour sum a of the forward
// iterate's z * n, z, n, b, invA and gz, the updates of gh, gb and ginv, and
// gg; the Huber mask is hfbs_step's.  hfbs_finish_adj: gz after the neighbour
// sum of gw = hfbs_adj_product.
__device__ __forceinline__ void hfbs_step_adj(float a, float z, float n, float b, float ia,
                                              float gz, float lambda, float alpha, float beta,
                                              float& gh, float& gb, float& ginv, float& gg) {
  const float t = __fmaf_rn(__fmul_rn(lambda, n), a, b);
  const float grad = __fmaf_rn(-t, ia, z);
  const float u = __fmaf_rn(-alpha, gz, gh);
  const float m = fabsf(grad) >= 1.345f ? 0.f : u;
  gh = __fmul_rn(beta, u);
  gb = __fmaf_rn(-ia, m, gb);
  ginv = __fmaf_rn(-t, m, ginv);
  gg = m;
}
__device__ __forceinline__ float hfbs_adj_product(float n, float ia, float gg) {
  return __fmul_rn(__fmul_rn(n, ia), gg);
}
__device__ __forceinline__ float hfbs_finish_adj(float gz, float gg, float n, float a,
                                                 float lambda) {
  return __fadd_rn(gz, __fmaf_rn(-__fmul_rn(lambda, n), a, gg));
}

// Solver parameters shared by a batch (HFBSGridParams minus the grid dims).
struct HParams {
  float sigma_x, sigma_y, sigma_l, lambda, alpha, beta;
  int bistoch_iter_max, optim_iter_max;
  float neg_exp_beta;
};

// Forward iterates kept for the HFBS adjoint, and its scratch grids (all
// total_voxels floats per plane).  segment 1: z_k (0 <= k < K) in hist plane
// k, nothing is recomputed.  segment S > 1: z and h at the start of every
// S-step segment go to slot j of ckz / ckh (step j*S), and the backward
// recomputes a segment's iterates into seg (S - 1 planes) with h ping-ponging
// through hrec / hrec2.  The adjoint's scratch: gz, gh, gb, ginv and two
// (gg, gw) pairs.
struct HfbsGradState {
  int segment = 1;
  float* hist = nullptr;
  float *ckz = nullptr, *ckh = nullptr, *seg = nullptr, *hrec = nullptr, *hrec2 = nullptr;
  float *gz = nullptr, *gh = nullptr, *gb = nullptr, *ginv = nullptr;
  float *gg = nullptr, *gw = nullptr, *gg2 = nullptr, *gw2 = nullptr;
};

// Grid planes of an HfbsGradState for K steps and segment S.
inline long long hfbs_grad_planes(int K, int S) {
  if (S == 1) return 8 + (K > 0 ? K : 0);
  const long long nck = (K + S - 1) / S;
  return 8 + 2 * nck + (S - 1) + 2;
}

// Point G's planes into an arena of hfbs_grad_planes(K, S) * tv floats.
inline void hfbs_carve_grad(HfbsGradState& G, float* arena, int K, int S, long long tv) {
  float* q = arena;
  auto take = [&](long long planes) {
    float* r = q;
    q += planes * tv;
    return r;
  };
  G = HfbsGradState{};
  G.segment = S;
  G.gz = take(1);
  G.gh = take(1);
  G.gb = take(1);
  G.ginv = take(1);
  G.gg = take(1);
  G.gw = take(1);
  G.gg2 = take(1);
  G.gw2 = take(1);
  if (S == 1) {
    G.hist = take(K > 0 ? K : 0);
  } else {
    const long long nck = (K + S - 1) / S;
    G.ckz = take(nck);
    G.ckh = take(nck);
    G.seg = take(S - 1);
    G.hrec = take(1);
    G.hrec2 = take(1);
  }
}

// Device buffers and sizes of a batch of HFBS instances.
struct HfbsBatch {
  const HInst* d_inst;
  int n_inst;
  // host copy of the instance table and the voxel budget of an L2-resident
  // group (0: all instances together); see hfbs_enqueue_solve
  const HInst* h_inst = nullptr;
  long long group_voxels = 0;
  // heavy-ball steps per launch: kHfbsMarchSteps (the march, where every
  // grid has at most kHfbsMarchMaxGL levels) or 1 (the one-step kernel for
  // every grid)
  int solve_steps = 4;
  // tensor maps of the grid planes for the marches' TMA loads (null: they
  // load by threads); owned by the caller, which
  // clears it when the instances' grids change
  TmaCache* tma = nullptr;
  // the bistochastized normalisation in n0 / n1 (by the parity of
  // bistoch_iter_max) is that of the same guide and grid: skip recomputing it
  bool reuse_norm = false;
  long long max_voxels, max_pixels, max_cells, max_lines;
  // voxels of the whole grid arena (instances and the gaps that round each
  // instance's grid to 32 voxels): the span of the elementwise kernels
  long long total_voxels;
  long long max_rows;  // max over instances of gy * gl (grid rows along x)
  int max_gl;
  const uchar4* guide;
  const void* target;  // storage type st
  const void* conf;
  Storage st;
  float* out;
  float *count, *csum, *b, *n0, *n1, *invA, *z0, *z1, *h, *t0, *t1, *t2, *ovf;
  float2* sgrid;  // the instances' slice grids (HInst::slice_off)
  // optional debug copies (single-instance class API)
  bool keep_debug;
  float* dbg_z_init;  // a copy of the first iterate (keep_debug)
  // non-null: record the forward iterates for hfbs_enqueue_backward (all
  // instances as one group)
  const HfbsGradState* grad = nullptr;
};

// ---- the marching kernels (hfbs_march.cu) -------------------------------------
// Levels a grid may have for them, and steps per pass over the grid.
constexpr int kHfbsMarchMaxGL = 64;
constexpr int kHfbsMarchSteps = 4;
// How the instances [first, first + count) are cut into blocks.
struct HfbsMarchPlan {
  int first = 0, count = 0, warps = 1, rows = 1, ahead = 1;
  unsigned blocks = 1;  // per instance, at most
};
HfbsMarchPlan hfbs_march_plan(const HfbsBatch& B, int first, int count);
// `steps` (1 .. kHfbsMarchSteps) heavy-ball steps of the plan's instances from
// (zs, hs) to (zd, hd), other buffers; rec: z after each of the first
// rec_steps steps, plane stride total_voxels.
int hfbs_march_solve(const HfbsBatch& B, const HfbsMarchPlan& P, const HParams& p,
                     const float* norm, const float* zs, float* zd, const float* hs, float* hd,
                     int steps, float* rec, int rec_steps, cudaStream_t s);
// `steps` bistochastization iterations from src to dst; it0: index of the
// first one (its parity is the pad faces' value).
int hfbs_march_bistoch(const HfbsBatch& B, const HfbsMarchPlan& P, const float* src, float* dst,
                       int it0, int steps, cudaStream_t s);
// ---- grids that stay on chip (hfbs_cluster.cu) ---------------------------------
struct HfbsClusterPlan {
  int size = 0;  // CTAs of an instance's cluster; 0: the instances do not fit
  int items = 0, threads = 0, first = 0, count = 0;
  size_t smem = 0;
};
// The cluster that holds each of the instances [first, first + count), or
// size 0.
HfbsClusterPlan hfbs_cluster_plan(const HfbsBatch& B, int first, int count);
// Any number of heavy-ball steps in one launch, bit for bit
// hfbs_march_solve's; hd null: h is not wanted.
int hfbs_cluster_solve(const HfbsBatch& B, const HfbsClusterPlan& P, const HParams& p,
                       const float* norm, const float* zs, float* zd, const float* hs, float* hd,
                       int steps, float* rec, int rec_steps, cudaStream_t s);
// All `steps` bistochastization iterations, from ones, into dst.
int hfbs_cluster_bistoch(const HfbsBatch& B, const HfbsClusterPlan& P, float* dst, int steps,
                         cudaStream_t s);
// The cluster that holds the adjoint of each instance, or size 0 (it keeps
// twice the registers a voxel), and the adjoint of all `steps` steps from the
// kept iterates z_k (plane k of hist): gz in place, gb and ginv written.
HfbsClusterPlan hfbs_cluster_adj_plan(const HfbsBatch& B);
int hfbs_cluster_adjoint(const HfbsBatch& B, const HfbsClusterPlan& P, const HParams& p,
                         const float* norm, const float* hist, float* gz, float* gb, float* ginv,
                         int steps, cudaStream_t s);
// Builds the tensor maps of grid planes (before a capture).
void hfbs_march_prepare(const HfbsBatch& B, const std::vector<const float*>& planes,
                        cudaStream_t s);

// Enqueue the whole HFBS::Optimize sequence (splat .. slice) on a stream.
int hfbs_enqueue_solve(const HfbsBatch& B, const HParams& p, cudaStream_t s,
                       const float** z_final = nullptr);

// Builds the grid tensor maps the solve of B will stage from (grid planes
// b, invA, both z and h buffers, both normalisation buffers, the counts),
// so that a graph capture of the solve finds them; a no-op without B.tma.
void hfbs_prepare_tma(const HfbsBatch& B, const HParams& p, cudaStream_t s);

// CTAs of the marching kernels that gave up waiting for their TMA loads since
// the library was loaded (0 on a healthy run).
unsigned long long hfbs_wait_timeouts();

// Whether the batch's heavy-ball steps and normalisation march (every grid
// at most kHfbsMarchMaxGL levels, host instance table given, solve_steps not
// 1).  The march's neighbour sums add rounded z * n products; the one-step
// kernel's fuse them (FMA).
bool hfbs_uses_march(const HfbsBatch& B);

// `steps` heavy-ball steps of every instance from (zs, hs) to (zd, hd): one
// march (steps <= kHfbsMarchSteps), else one one-step launch (steps == 1, h
// updated in place in hd: the caller passes hs == hd).  rec: z after each of
// the first rec_steps steps, plane stride total_voxels (marches only).
int hfbs_launch_steps(const HfbsBatch& B, const HParams& p, const float* norm,
                      const float* zs, float* zd, const float* hs, float* hd, int steps,
                      float* rec, int rec_steps, cudaStream_t s);

// X -> Y -> Z Laplace blur of two grids s0, s1 into x0, x1 (y0, y1 scratch).
void hfbs_launch_blur_pair(const HfbsBatch& B, const HParams& p, const float* s0,
                           const float* s1, float* x0, float* x1, float* y0, float* y1,
                           cudaStream_t s);

// Adjoint of the last hfbs_enqueue_solve of B (run with B.grad): upstream
// gradient gout (pixel layout of the instances) to dL/dtarget and
// dL/dconfidence (same layout; either may be null).
int hfbs_enqueue_backward(const HfbsBatch& B, const HParams& p, const float* gout,
                          float* grad_t, float* grad_c, cudaStream_t s);

}  // namespace dtsgb
