// The iterative HFBS stages as time-skewed marches over the grid: several
// heavy-ball steps (src/hfbs.cu:201-239) or bistochastization iterations
// (src/hfbs.cu:126-155) per pass over memory, for grids of up to 64 levels.
//
// A warp holds 32 neighbouring columns x (lane = x) of four levels, a CTA the
// ceil(gl / 4) warps of all levels, and the CTA marches along y.  When plane
// y of the input arrives, step 1 updates plane y - 1, step 2 plane y - 2, ...,
// step K plane y - K: the neighbours of a voxel along y are values its own
// thread has just produced, those along l are in the same thread but for the
// ends of its four levels, and those along x come by warp shuffle.  Nothing
// is recomputed along y and l, and 24 of the 32 columns are useful along x.
// (A thread per column of a 24 x 24 block, the form this replaces, reads four
// neighbours and b and invA from shared memory per voxel and step, uses 44%
// of the columns and holds at most 16 levels.)  Measured per heavy-ball step:
// 57.5 us by one-step passes and 18 so on a 408 x 306 x 64 grid, 52 us in
// blocks and 40 so on 64 grids of 16 levels (11.85 M voxels in all); per
// bistochastization iteration 81 and 33, 62 and 39.
//
// Per plane: the five planes z, h, n, b, invA (two for the normalisation)
// arrive by TMA in a ring, one plane ahead of their use; a thread reads only
// its own entries.  n, b and invA stay in the ring for the K steps that use
// them; z, h and the z * n of three planes per step are registers.  One
// barrier per plane: the ends of the four levels (z * n of the next plane's
// centre) cross it through a double-buffered exchange.
//
// Bound by dependent instructions at 16 warps an SM, which take every register
// (issue slots 74% busy at 64 levels, 46% at 16): about 34 instructions per
// voxel and step, 13 of them floating point, 2 shuffles, 4 shared-memory reads
// and 10 moves and selects; memory traffic is 28 B a voxel and pass, a quarter
// of the DRAM's rate.
//
// Outside the grid and above level gl everything is zero (the TMA fill), so
// z * n adds zero to a neighbour sum there; those voxels are never updated.
// Sums are added in the reference's order (x-1, x+1, y-1, y+1, l-1, l+1) over
// rounded products.
#include <algorithm>
#include <vector>

#include "../../include/dtsgb.h"
#include "dtsgb_internal.cuh"
#include "hfbs_internal.cuh"
#include "tma.cuh"

namespace dtsgb {
namespace {

constexpr int kV = 4;                                    // levels a thread
constexpr int kBoxX = 32;                                // lanes
// Columns a strip is responsible for: lanes kPad .. kPad + kUse - 1 are at
// least kHfbsMarchSteps inside the box, and its first column (24 i - 4) is a
// multiple of four, as a TMA load's innermost coordinate must be.
constexpr int kPad = 4, kUse = 24;
static_assert(kPad >= kHfbsMarchSteps && kPad % 4 == 0 && kUse % 4 == 0 &&
                  kBoxX - kPad - kUse >= kHfbsMarchSteps,
              "halo of a strip");

// Planes requested ahead where few blocks leave their SMs idle between planes
// (a plane step then takes less than a TMA load does), one otherwise.
constexpr int kAhead = 3;

__device__ unsigned long long g_wait_timeouts = 0;

struct MarchMaps {
  const CUtensorMap *z, *h, *n, *b, *a;  // normalisation: z the input, n the counts
};
struct MarchArgs {
  const float *z, *h, *n, *b, *a;  // the same planes (loads without tensor maps)
  float *zd, *hd;
  float* rec;  // z after step k + 1 in plane k, stride rec_stride, rec_steps of them
  long long rec_stride;
  int rec_steps;
  float lambda, alpha, beta;
  int it0;   // normalisation: index of the pass's first iteration
  int rows;  // planes per block along y
};

enum { kHeavyBall = 0, kBistoch = 1 };

// Floats of shared memory: the ring (the planes the K steps use, the newest
// and D arriving), the inputs of step 1, the exchange.
template <int MODE, int K, int D>
__host__ __device__ constexpr int smem_floats(int nw) {
  const int pl = nw * kV * kBoxX;
  return pl * ((MODE == kHeavyBall ? 3 : 1) * (K + 1 + D) +
               (MODE == kHeavyBall ? 2 : 1) * (D + 1)) +
         K * 2 * 2 * nw * 32;
}
template <int MODE, int K, int D>
constexpr size_t smem_bytes(int nw) {
  return sizeof(float) * smem_floats<MODE, K, D>(nw) + 8 * (D + 1);
}

// D: planes requested ahead of the one in use.
template <int MODE, bool REC, int K, int D>
__global__ void __launch_bounds__(MODE == kBistoch ? 640 : 512, 1)
    k_hfbs_march(const HInst* __restrict__ insts, MarchArgs A, MarchMaps m) {
  pdl_wait_then_release();  // launched as a dependent of the previous pass
  constexpr int NR = MODE == kHeavyBall ? 3 : 1;  // arrays in the ring
  constexpr int NI = MODE == kHeavyBall ? 2 : 1;  // inputs of step 1
  constexpr int SL = K + 1 + D, NB = D + 1;       // ring slots; input slots
  extern __shared__ __align__(128) float sm[];
  const HInst I = insts[blockIdx.y];
  const int gx = I.gx, gy = I.gy, gl = I.gl;
  const int strips = (gx + kUse - 1) / kUse;
  const int seg = blockIdx.x / strips, strip = blockIdx.x - seg * strips;
  const int y0 = seg * A.rows;
  if (y0 >= gy) return;
  const int y1 = min(y0 + A.rows, gy);
  const int nw = blockDim.x >> 5, PL = nw * kV * kBoxX;
  float* ring = sm;                          // [SL][NR][PL]
  float* inp = ring + SL * NR * PL;          // [NB][NI][PL]
  float* ex = inp + NB * NI * PL;            // [2][K][2][nw][32]
  unsigned long long* bar =
      reinterpret_cast<unsigned long long*>(ex + K * 2 * 2 * nw * 32);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int x0 = strip * kUse - kPad, x = x0 + lane;
  const bool inx = x >= 0 && x < gx;
  const int ya = y0 - K, N = y1 - y0 + 2 * K;  // input planes ya .. ya + N - 1
  const int plane = I.px * gy;
  const int own = (w * kV) * kBoxX + lane;     // this thread's entry of a plane
  const long long gcol = I.grid_off + (long long)(w * kV) * plane + x;  // + y * px
  const bool use_tma = m.z != nullptr && (smem_u32(sm) & 127u) == 0;
  bool in[kV];  // inside the grid (along x and l)
#pragma unroll
  for (int v = 0; v < kV; ++v) in[v] = inx && w * kV + v < gl;
  // input plane j (0 .. N - 1) into ring slot rs and input slot is: by TMA from
  // thread 0, else every thread its own entries (zero outside the grid)
  auto request = [&](int j, int rs, int is) {
    float* zi = inp + is * NI * PL;
    float* r = ring + rs * NR * PL;
    const int y = ya + j;
    if (use_tma) {
      if (tid == 0) {
        unsigned long long* bj = bar + is;
        mbar_arrive_expect_tx(bj, (unsigned)(sizeof(float) * PL * (NR + NI)));
        tma_load_3d(zi, m.z + blockIdx.y, x0, y, 0, bj);
        tma_load_3d(r, m.n + blockIdx.y, x0, y, 0, bj);
        if (MODE == kHeavyBall) {
          tma_load_3d(zi + PL, m.h + blockIdx.y, x0, y, 0, bj);
          tma_load_3d(r + PL, m.b + blockIdx.y, x0, y, 0, bj);
          tma_load_3d(r + 2 * PL, m.a + blockIdx.y, x0, y, 0, bj);
        }
      }
    } else {
#pragma unroll
      for (int v = 0; v < kV; ++v) {
        const bool ok = in[v] && y >= 0 && y < gy;
        const long long g = ok ? gcol + (long long)v * plane + (long long)y * I.px : 0;
        const int o = own + v * kBoxX;
        zi[o] = ok ? A.z[g] : 0.f;
        r[o] = ok ? A.n[g] : 0.f;
        if (MODE == kHeavyBall) {
          zi[PL + o] = ok ? A.h[g] : 0.f;
          r[PL + o] = ok ? A.b[g] : 0.f;
          r[2 * PL + o] = ok ? A.a[g] : 0.f;
        }
      }
    }
  };
  if (tid == 0) {
#pragma unroll
    for (int k = 0; k < NB; ++k) mbar_init(&bar[k], 1);
    mbar_fence_init();
  }
  for (int i = tid; i < K * 2 * 2 * nw * 32; i += blockDim.x) ex[i] = 0.f;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NB; ++k)
    if (k < N) request(k, k, k);
  // stage k (index k - 1): z, h and z * n of its plane, z * n of the plane
  // before; the normalisation's v is its own z * n
  float zc[K][kV], hc[K][kV], pm[K][kV], pc[K][kV];
#pragma unroll
  for (int k = 0; k < K; ++k)
#pragma unroll
    for (int v = 0; v < kV; ++v) zc[k][v] = hc[k][v] = pm[k][v] = pc[k][v] = 0.f;
  // the pad faces of the normalisation: 1 on even iterations, 0 on odd ones
  auto pad_at = [&](int it) -> float { return (it & 1) ? 0.f : 1.f; };
  const bool face_x = MODE == kBistoch && I.cov_x && x == gx;
  const bool face_y = MODE == kBistoch && I.cov_y && inx;
  const bool out_lane = inx && lane >= kPad && lane < kPad + kUse;
  const int ex_lo = (nw + max(w, 1) - 1) * 32 + lane, ex_hi = min(w + 1, nw - 1) * 32 + lane;
  const bool has_lo = w > 0, has_hi = w + 1 < nw;
  int slot = 0, is = 0;       // j % SL, j % NB
  unsigned parity = 0;        // of input slot `is`: flips when it wraps
  // (by two: half of the moves between planes are renamings; 3% of a solve.  The
  // normalisation does without and fits five blocks of four warps an SM.)
#pragma unroll (REC || MODE == kBistoch ? 1 : 2)
  for (int j = 0; j < N; ++j) {
    const bool got = !use_tma || mbar_wait_bounded(&bar[is], parity, kTmaWaitPolls);
    const float* zi = inp + is * NI * PL + own;
    const float* ri = ring + slot * NR * PL + own;
    const float* exr = ex + (j & 1) * (K * 2 * nw * 32);
    const int yj = ya + j;
    float cz[kV], ch[kV], cp[kV];  // the newest plane of the step before
#pragma unroll
    for (int v = 0; v < kV; ++v) {
      cz[v] = zi[v * kBoxX];
      ch[v] = MODE == kHeavyBall ? zi[PL + v * kBoxX] : 0.f;
      if (MODE == kHeavyBall) {
        cp[v] = __fmul_rn(cz[v], ri[v * kBoxX]);
      } else {
        const bool face = (face_x && yj >= 0 && yj < gy) || (face_y && yj == gy);
        cp[v] = face && w * kV + v < gl ? pad_at(A.it0) : cz[v];
      }
    }
    // Stages have no branches (a branch's merge costs a register move per
    // value): before j = 2k a stage computes on planes that no later stage's
    // valid planes read, and outside the grid on zeros, which stay zeros.
#pragma unroll
    for (int k = 1; k <= K; ++k) {
      const int y = yj - k;
      const bool iny = (unsigned)y < (unsigned)gy;
      float nz[kV], nh[kV], np[kV];
      float (&P)[kV] = pc[k - 1];
      int sk = slot - k;
      if (sk < 0) sk += SL;
      const float* rk = ring + sk * NR * PL + own;
      const float* e = exr + (k - 1) * (2 * nw * 32);
      const float lo = has_lo ? e[ex_lo] : 0.f;
      const float hi = has_hi ? e[ex_hi] : 0.f;
#pragma unroll
      for (int v = 0; v < kV; ++v) {
        const float below = v > 0 ? P[v > 0 ? v - 1 : 0] : lo;
        float above = v + 1 < kV ? P[v + 1 < kV ? v + 1 : v] : hi;
        const float xm = __shfl_up_sync(0xffffffffu, P[v], 1);
        const float xp = __shfl_down_sync(0xffffffffu, P[v], 1);
        if (MODE == kHeavyBall) {
          const float n = rk[v * kBoxX];
          nz[v] = zc[k - 1][v];
          nh[v] = hc[k - 1][v];
          hfbs_step(xm, xp, pm[k - 1][v], cp[v], below, above, n, rk[PL + v * kBoxX],
                    rk[2 * PL + v * kBoxX], A.lambda, A.alpha, A.beta, nz[v], nh[v]);
          np[v] = __fmul_rn(nz[v], n);
        } else {
          if (w * kV + v + 1 == gl) above = I.cov_l ? pad_at(A.it0 + k - 1) : 0.f;
          float a = xm;
          a += xp;
          a += pm[k - 1][v];
          a += cp[v];
          a += below;
          a += above;
          const float vc = P[v];
          const float blurred = 2.f * vc + a;
          // where nothing is computed the operands are 1: zeros and what
          // stands in unused memory would take the slow division and root
          const bool ok = in[v] && iny && j >= 2 * k;
          const float num = ok ? vc * (rk[v * kBoxX] + 0.00001f) : 1.f;
          const float den = ok ? blurred + 0.00001f : 1.f;
          nz[v] = __fsqrt_rn(__fdiv_rn(num, den));
          nh[v] = 0.f;
          const bool face = ((face_x && iny) || (face_y && y == gy)) && w * kV + v < gl;
          np[v] = ok ? nz[v] : face ? pad_at(A.it0 + k) : 0.f;
        }
      }
      // outputs of every step when recorded
      if (REC && k <= A.rec_steps && j >= 2 * k && y >= y0 && y < y1 && out_lane) {
        float* o = A.rec + (k - 1) * A.rec_stride + gcol + (long long)y * I.px;
#pragma unroll
        for (int v = 0; v < kV; ++v)
          if (in[v]) o[(long long)v * plane] = nz[v];
      }
#pragma unroll
      for (int v = 0; v < kV; ++v) {
        pm[k - 1][v] = pc[k - 1][v];
        pc[k - 1][v] = cp[v];
        if (MODE == kHeavyBall) {
          zc[k - 1][v] = cz[v];
          hc[k - 1][v] = ch[v];
        }
        cz[v] = nz[v];
        ch[v] = nh[v];
        cp[v] = np[v];
      }
    }
    // the last stage's plane
    if (j >= 2 * K && out_lane) {  // y0 <= yj - K < y1 for these j
      const long long g = gcol + (long long)(yj - K) * I.px;
#pragma unroll
      for (int v = 0; v < kV; ++v)
        if (in[v]) {
          A.zd[g + (long long)v * plane] = MODE == kHeavyBall ? cz[v] : cp[v];
          if (MODE == kHeavyBall) A.hd[g + (long long)v * plane] = ch[v];
        }
    }
    // the ends of the next plane's centres
    float* exw = ex + ((j + 1) & 1) * (K * 2 * nw * 32) + w * 32 + lane;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      exw[k * (2 * nw * 32)] = pc[k][0];
      exw[k * (2 * nw * 32) + nw * 32] = pc[k][kV - 1];
    }
    if (__syncthreads_or(!got)) {  // a wait ran out: recorded, and the block gives up
      if (tid == 0) atomicAdd(&g_wait_timeouts, 1ull);
      for (int k = j; k < min(j + NB, N); ++k)  // the copies in flight may still land
        (void)mbar_wait_bounded(&bar[k % NB], (k / NB) & 1, kTmaWaitPolls);
      return;
    }
    if (j + NB < N) {
      if (use_tma && tid == 0) fence_proxy_async_shared();
      request(j + NB, slot + NB >= SL ? slot + NB - SL : slot + NB, is);
    }
    if (++slot == SL) slot = 0;
    if (++is == NB) {
      is = 0;
      parity ^= 1u;
    }
  }
}

template <int MODE, bool REC, int K, int D>
int launch(const HfbsBatch& B, const HfbsMarchPlan& P, const MarchArgs& A, const MarchMaps& m,
           cudaStream_t s) {
  const size_t smem = smem_bytes<MODE, K, D>(P.warps);
  auto kern = k_hfbs_march<MODE, REC, K, D>;
  DTSGB_CUDA(allow_smem(kern, smem));
  DTSGB_CUDA(launch_dependent(kern, dim3(P.blocks, P.count), dim3(P.warps * 32), smem, s,
                              B.d_inst + P.first, A, m));
  return DTSGB_OK;
}

template <int MODE, bool REC>
int launch_steps(const HfbsBatch& B, const HfbsMarchPlan& P, int steps, const MarchArgs& A,
                 const MarchMaps& m, cudaStream_t s) {
  switch (steps) {
    case 1: return launch<MODE, REC, 1, 1>(B, P, A, m, s);
    case 2: return launch<MODE, REC, 2, 1>(B, P, A, m, s);
    case 3: return launch<MODE, REC, 3, 1>(B, P, A, m, s);
  }
  return P.ahead > 1 ? launch<MODE, REC, kHfbsMarchSteps, kAhead>(B, P, A, m, s)
                     : launch<MODE, REC, kHfbsMarchSteps, 1>(B, P, A, m, s);
}

// The table of tensor maps of grid plane `plane` over B's instances (boxes of
// 32 columns, one row and all levels), or null.
std::vector<TmaGrid> tma_grids(const HfbsBatch& B) {
  std::vector<TmaGrid> g(B.n_inst);
  for (int i = 0; i < B.n_inst; ++i) {
    const HInst& H = B.h_inst[i];
    g[i] = TmaGrid{H.grid_off, H.gx, H.gy, H.gl, H.px};
  }
  return g;
}
const CUtensorMap* grid_map(const HfbsBatch& B, const float* plane, cudaStream_t s) {
  if (!B.tma || !B.h_inst) return nullptr;
  const std::vector<TmaGrid> g = tma_grids(B);
  return B.tma->get_grid(g.data(), B.n_inst, plane, kBoxX, 1, (B.max_gl + kV - 1) / kV * kV, s);
}

}  // namespace

unsigned long long hfbs_wait_timeouts() {
  unsigned long long v = 0;
  if (cudaMemcpyFromSymbol(&v, g_wait_timeouts, sizeof v) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return v;
}

void hfbs_march_prepare(const HfbsBatch& B, const std::vector<const float*>& planes,
                        cudaStream_t s) {
  if (!B.tma || !B.h_inst) return;
  const std::vector<TmaGrid> g = tma_grids(B);
  B.tma->prepare_grids(g.data(), B.n_inst, planes, kBoxX, 1, (B.max_gl + kV - 1) / kV * kV, s);
}

// Planes per block: the choice with the least modelled time.  A block of
// `warps` warps takes rows + 2K + 4 plane steps (4: its first loads); a plane
// step takes the larger of its latency and of the issue time of the blocks
// that share the SM.
HfbsMarchPlan hfbs_march_plan(const HfbsBatch& B, int first, int count) {
  constexpr int K = kHfbsMarchSteps;
  HfbsMarchPlan P;
  P.first = first;
  P.count = count;
  P.warps = (B.max_gl + kV - 1) / kV;
  int max_gy = 1;
  for (int i = 0; i < count; ++i) max_gy = std::max(max_gy, B.h_inst[first + i].gy);
  // SMs and blocks an SM holds (128 registers a thread; shared memory)
  constexpr int sms = 152, sm_smem = 228 * 1024;
  const int smem = (int)smem_bytes<kHeavyBall, K, 1>(P.warps) + 1024;
  const int per_sm = std::max(1, std::min(16 / P.warps, sm_smem / smem));
  const double latency = 600.0, issue = 30.0 * K * P.warps;
  double best = -1.0;
  long long blocks = 1;
  for (int segs = 1, last = 0; segs <= max_gy; ++segs) {
    const int rows = (max_gy + segs - 1) / segs;
    if (rows == last) continue;
    last = rows;
    if (rows < 4 && best >= 0) break;
    long long total = 0, most = 1;
    for (int i = 0; i < count; ++i) {
      const HInst& H = B.h_inst[first + i];
      const long long t =
          (long long)((H.gx + kUse - 1) / kUse) * ((H.gy + rows - 1) / rows);
      total += t;
      most = std::max(most, t);
    }
    const long long a = (total + sms - 1) / sms;
    const long long full = a / per_sm, rest = a % per_sm;
    const double cost = (rows + 2 * K + 4) *
                        ((double)full * std::max(latency, per_sm * issue) +
                         (rest ? std::max(latency, rest * issue) : 0.0));
    if (best < 0 || cost < best) {
      best = cost;
      P.rows = rows;
      P.blocks = (unsigned)most;
      blocks = total;
    }
  }
  P.ahead = blocks <= 2 * sms && smem_bytes<kHeavyBall, K, kAhead>(P.warps) <= kMaxSmem ? kAhead : 1;
  return P;
}

int hfbs_march_solve(const HfbsBatch& B, const HfbsMarchPlan& P, const HParams& p,
                     const float* norm, const float* zs, float* zd, const float* hs, float* hd,
                     int steps, float* rec, int rec_steps, cudaStream_t s) {
  const float* planes[5] = {zs, hs, norm, B.b, B.invA};
  const CUtensorMap* t[5];
  bool all = true;
  for (int k = 0; k < 5; ++k) all = (t[k] = grid_map(B, planes[k], s)) && all;
  const int f = P.first;
  const MarchMaps m =
      all ? MarchMaps{t[0] + f, t[1] + f, t[2] + f, t[3] + f, t[4] + f} : MarchMaps{};
  const MarchArgs A{zs, hs, norm, B.b, B.invA, zd, hd, rec, B.total_voxels, rec_steps,
                    p.lambda, p.alpha, p.beta, 0, P.rows};
  return rec_steps > 0 ? launch_steps<kHeavyBall, true>(B, P, steps, A, m, s)
                       : launch_steps<kHeavyBall, false>(B, P, steps, A, m, s);
}

int hfbs_march_bistoch(const HfbsBatch& B, const HfbsMarchPlan& P, const float* src, float* dst,
                       int it0, int steps, cudaStream_t s) {
  const CUtensorMap* ms = grid_map(B, src, s);
  const CUtensorMap* mc = ms ? grid_map(B, B.count, s) : nullptr;
  const MarchMaps m = mc ? MarchMaps{ms + P.first, nullptr, mc + P.first, nullptr, nullptr}
                         : MarchMaps{};
  const MarchArgs A{src, nullptr, B.count, nullptr, nullptr, dst, nullptr, nullptr, 0, 0,
                    0.f, 0.f, 0.f, it0, P.rows};
  return launch_steps<kBistoch, false>(B, P, steps, A, m, s);
}

}  // namespace dtsgb
