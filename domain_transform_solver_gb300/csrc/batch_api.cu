// Batched DTS / HFBS over many images of uneven size (C ABI in
// include/dtsgb.h).  All instances live in one arena: plane k of instance i
// starts at element offset off_i (rows pitched to 32 elements), and every
// kernel launch covers every instance through the instance and tile tables,
// so a solve costs the same number of launches for 1 or 1000 images.  The
// fixed launch sequence of each solve can be captured as a CUDA graph and
// replayed (the iteration counts are fixed and nothing depends on data).
//
// HFBS instances of a batch behave like HFBS objects whose max grid exceeds
// their grid on every axis (as in the reference's CLIs): pad faces of axes
// with g % 8 != 0 are covered, and the luma-overflow plane is stored.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <fstream>
#include <initializer_list>
#include <map>
#include <sstream>
#include <string>
#include <vector>

#include "../../include/dtsgb.h"
#include "color.cuh"
#include "dtsgb_internal.cuh"
#include "hfbs_internal.cuh"
#include "tma.cuh"

using namespace dtsgb;

namespace {

struct Graph {
  cudaGraphExec_t exec = nullptr;
  std::vector<char> key;
};

template <typename T>
void key_append(std::vector<char>& k, const T& v) {
  const char* p = reinterpret_cast<const char*>(&v);
  k.insert(k.end(), p, p + sizeof(T));
}

enum { HG_COUNT = 0, HG_CSUM, HG_B, HG_N0, HG_N1, HG_INVA, HG_Z0, HG_Z1, HG_H,
       HG_T0, HG_T1, HG_T2, HG_NUM };

}  // namespace

struct dtsgb_batch_s {
  int n = 0;
  unsigned flags = 0;
  Storage st = Storage::F32;
  int ref_y = 1;
  std::vector<Inst> inst;
  long long total = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  uchar4* guide = nullptr;
  void* target = nullptr;
  void* conf = nullptr;
  uint32_t* bounds = nullptr;
  float* v[2] = {nullptr, nullptr};
  float* hout = nullptr;
  // host uploads: every image is copied whole (one contiguous copy per
  // plane) into a dense staging area, then one kernel writes the pitched
  // planes; soff[i] = pixels of the instances before i
  std::vector<long long> soff;
  long long dense = 0;
  long long* d_soff = nullptr;
  unsigned char* stage = nullptr;  // dense x (rgba 4 B, target 4 B, conf 4 B)
  Inst* d_inst = nullptr;
  // blocks of the DTS passes per halo (several instances only), carved from
  // pass_mem; kept until the batch is destroyed (ensure_pass_blocks)
  struct PassTables {
    Tile *x = nullptr, *y = nullptr;
    unsigned nx = 0, ny = 0;
  };
  std::map<int, PassTables> pass;
  std::vector<Tile*> pass_mem;
  size_t pass_room = 0, pass_left = 0;  // blocks of an allocation, left in the last one
  bool small = false;               // accepted and returned (DTSGB_TUNE_DTS_TILE)
  long long hfbs_group_voxels = 0;  // L2-resident HFBS group budget (0: off)
  int hfbs_solve_steps = 4;         // heavy-ball steps per launch (4 or 1)
  int bounds_seg = 8;               // accepted and returned (DTSGB_TUNE_BOUNDS_SEGMENT)
  // Guide-derived state kept across solves while the guide is unchanged
  // (video frames that change only the target): the DTS window bounds and
  // the HFBS bistochastized normalisation.
  unsigned long long guide_gen = 0;  // bumped by every guide upload
  bool reuse = true;
  struct BoundsKey {
    unsigned long long gen;
    float rx, ry, sz;
    int ref_y;
  } bkey{~0ull, 0.f, 0.f, 0.f, 0};
  struct NormKey {
    unsigned long long gen;
    float sx, sy, sl;
    int bistoch;
  } nkey{~0ull, 0.f, 0.f, 0.f, 0};
  int dts_res = -1;
  bool hfbs_done = false;
  bool use_graphs = true;
  Graph g_dts, g_hfbs;
  std::vector<HInst> hinst;
  HInst* d_hinst = nullptr;
  float* hg[HG_NUM] = {};
  long long gcap = 0;
  float* ovf = nullptr;
  long long ocap = 0;
  float2* sgrid = nullptr;
  long long scap = 0;
  // gradients of the DTS solve
  bool grad = false;
  int grad_seg_req = 0;          // 0: dts_checkpoint_segment(N)
  int grad_seg = 1;              // segment length of the planes below
  int grad_n = -1;               // iterations the adjoint replays (-1: none kept)
  std::vector<float*> gplanes;   // checkpoints, segment planes, 2 adjoint, dt, dc
  dtsgb_optimize_params gopt{};  // parameters of the solve the planes belong to
  float ghalo = 0.f;
  Graph g_bwd;
  // gradients of the HFBS solve (the same enable_grad switch): the kept
  // iterates and adjoint grids (hfbs_grad_planes) in hgbuf; three pixel
  // planes (dL/dout, dL/dtarget, dL/dconfidence) in hpix
  float* hgbuf = nullptr;
  size_t hgcap = 0;  // floats
  float* hpix = nullptr;
  HfbsGradState hgs{};
  int hgrad_seg = 0, hgrad_planes = 0;
  bool hgrad_ready = false;  // the last HFBS solve kept its iterates
  HfbsBatch hB{};            // that solve's batch description and parameters
  HParams hhp{};
  Graph g_hbwd;

  // tensor maps of the HFBS grid planes (cleared when the grids change)
  TmaCache htma;

  size_t tsize() const { return st == Storage::F32 ? 4 : 2; }
};

namespace {

void drop_graph(dtsgb_batch_t b, Graph& g) {
  if (g.exec) {
    cudaGraphExecDestroy(g.exec);
    g.exec = nullptr;
  }
  prof_drop_captured(&g);
  g.key.clear();
}

void free_grad_planes(dtsgb_batch_t b) {
  for (auto& p : b->gplanes) dfree(p);
  b->gplanes.clear();
}

void batch_free(dtsgb_batch_t b) {
  drop_graph(b, b->g_dts);
  drop_graph(b, b->g_hfbs);
  drop_graph(b, b->g_bwd);
  drop_graph(b, b->g_hbwd);
  free_grad_planes(b);
  dfree(b->hgbuf);
  dfree(b->hpix);
  dfree(b->guide);
  dfree(b->target);
  dfree(b->conf);
  dfree(b->bounds);
  dfree(b->v[0]);
  dfree(b->v[1]);
  dfree(b->hout);
  dfree(b->d_inst);
  for (Tile*& p : b->pass_mem) dfree(p);
  dfree(b->d_hinst);
  for (auto& p : b->hg) dfree(p);
  dfree(b->ovf);
  dfree(b->sgrid);
  dfree(b->d_soff);
  dfree(b->stage);
  if (b->own_stream && b->stream) cudaStreamDestroy(b->stream);
  b->stream = nullptr;
}

// Planes for the adjoint of an N-iteration solve with segment length seg:
// ceil(N/seg) - 1 checkpoints, seg recompute planes, two adjoint planes and
// the two gradient planes.  Reallocation drops the graphs that captured the
// old pointers.
int ensure_grad_planes(dtsgb_batch_t b, int n_iter, int seg) {
  const int nseg = (n_iter + seg - 1) / seg;
  const size_t need = (size_t)std::max(nseg - 1, 0) + seg + 4;
  if (b->gplanes.size() == need && b->grad_seg == seg) return DTSGB_OK;
  DTSGB_CUDA(cudaStreamSynchronize(b->stream));
  drop_graph(b, b->g_dts);
  drop_graph(b, b->g_bwd);
  free_grad_planes(b);
  b->grad_seg = seg;
  for (size_t k = 0; k < need; ++k) {
    float* p = nullptr;
    int st = dalloc(&p, (size_t)b->total);
    if (st) {
      free_grad_planes(b);
      return st;
    }
    b->gplanes.push_back(p);
  }
  return DTSGB_OK;
}

DtsGrad grad_view(dtsgb_batch_t b, int n_iter) {
  const int seg = b->grad_seg;
  const int ncp = std::max((n_iter + seg - 1) / seg - 1, 0);
  float* const* P = b->gplanes.data();
  DtsGrad G;
  G.seg = seg;
  G.cp = P;
  G.segbuf = P + ncp;
  G.g[0] = P[ncp + seg];
  G.g[1] = P[ncp + seg + 1];
  return G;
}
float* grad_plane_t(dtsgb_batch_t b) { return b->gplanes[b->gplanes.size() - 2]; }
float* grad_plane_c(dtsgb_batch_t b) { return b->gplanes[b->gplanes.size() - 1]; }

// Whether the caller is capturing the batch's stream (without graphs of the
// batch's own, which a capture refuses): what is enqueued runs at a replay.
bool callers_capture(dtsgb_batch_t b) {
  cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
  return !b->use_graphs && cudaStreamIsCapturing(b->stream, &c) == cudaSuccess &&
         c != cudaStreamCaptureStatusNone;
}

// Blocks of the passes over the whole batch for a halo.
dim3 pass_block_totals(dtsgb_batch_t b, int halo) {
  dim3 t(0, 0);
  for (const Inst& I : b->inst) {
    const dim3 c = dts_pass_block_counts(I, halo);
    t.x += c.x;
    t.y += c.y;
  }
  return t;
}

// The block tables of the DTS passes for a halo.  A graph that the caller has
// captured may hold their addresses, so they stay, and are not changed, until
// the batch is destroyed.  They are written by a kernel on the batch's stream
// into memory set aside at creation (a few halos' worth, more is allocated
// then): a solve with a halo of its own waits for nothing.  *fresh: written now.
int ensure_pass_blocks(dtsgb_batch_t b, int halo, bool* fresh) {
  *fresh = false;
  if (b->n == 1 || b->pass.count(halo)) return DTSGB_OK;
  cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
  DTSGB_CUDA(cudaStreamIsCapturing(b->stream, &c));
  if (c != cudaStreamCaptureStatusNone) return DTSGB_OK;  // a launch per instance then
  const dim3 n = pass_block_totals(b, halo);
  const size_t need = (size_t)n.x + n.y;
  if (need > b->pass_left) {
    const size_t room = std::max(need, b->pass_room);
    Tile* p = nullptr;
    const cudaError_t e = cudaMalloc((void**)&p, room * sizeof(Tile));
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      return e == cudaErrorMemoryAllocation
                 ? fail(DTSGB_ERR_OUT_OF_MEMORY, "cudaMalloc: out of memory")
                 : cuda_fail(e, "cudaMalloc");
    }
    b->pass_mem.push_back(p);
    b->pass_room = b->pass_left = room;
  }
  dtsgb_batch_s::PassTables t;
  t.x = b->pass_mem.back() + (b->pass_room - b->pass_left);
  t.y = t.x + n.x;
  t.nx = n.x;
  t.ny = n.y;
  if (int st = launch_pass_blocks(b->d_inst, b->inst.data(), b->n, halo, t.x, t.y, b->stream))
    return st;
  b->pass_left -= need;
  b->pass[halo] = t;
  *fresh = true;
  return DTSGB_OK;
}
DtsLaunch iter_launch(dtsgb_batch_t b, int halo) {
  DtsLaunch L{b->d_inst, nullptr, 0, b->n, false, nullptr, 0, b->inst.data()};
  const auto t = b->pass.find(halo);
  if (t == b->pass.end()) return L;
  L.d_xblocks = t->second.x;
  L.d_yblocks = t->second.y;
  L.n_xblocks = t->second.nx;
  L.n_yblocks = t->second.ny;
  return L;
}

// Run `enqueue` directly, or through the solve's CUDA graph (captured on the
// first call with this key, replayed afterwards).
template <typename F>
int run_graph(dtsgb_batch_t b, Graph& g, std::vector<char> key, F enqueue) {
  if (!b->use_graphs) return enqueue();
  key_append(key, prof_enabled());
  if (g.exec && g.key == key) {
    DTSGB_CUDA(cudaGraphLaunch(g.exec, b->stream));
    return DTSGB_OK;
  }
  drop_graph(b, g);
  prof_set_capture_tag(&g);
  cudaError_t e = cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeRelaxed);
  if (e != cudaSuccess) {
    prof_set_capture_tag(nullptr);
    return cuda_fail(e, "cudaStreamBeginCapture");
  }
  int st = enqueue();
  cudaGraph_t graph = nullptr;
  e = cudaStreamEndCapture(b->stream, &graph);
  prof_set_capture_tag(nullptr);
  if (st) {
    if (graph) cudaGraphDestroy(graph);
    prof_drop_captured(&g);
    return st;
  }
  if (e != cudaSuccess) return cuda_fail(e, "cudaStreamEndCapture");
  e = cudaGraphInstantiate(&g.exec, graph, 0);
  cudaGraphDestroy(graph);
  if (e != cudaSuccess) {
    g.exec = nullptr;
    prof_drop_captured(&g);
    return cuda_fail(e, "cudaGraphInstantiate");
  }
  g.key = key;
  DTSGB_CUDA(cudaGraphLaunch(g.exec, b->stream));
  return DTSGB_OK;
}

// ---- dense images <-> pitched planes -------------------------------------------
// Bound by HBM (12 B/px read, 8 or 12 written by an upload).  A block of 8
// warps takes kCopyRows rows x `cols` pixels of one instance, a warp per row:
// 512 columns (four rounds of loads a warp) for images that fill the SMs
// that way, else one round's 128, or 32 where single pixels are copied (a
// small image is latency: 333x250 loses 2 us a solve with four).  Four adjacent
// pixels per thread and 16-byte accesses where the dense rows allow them
// (the width a multiple of 4 and every pointer 16-byte aligned; the planes'
// rows always are), else four single pixels whose loads are issued before
// their stores.  With one pixel per thread and a block per row or five:
// 84 us at 3264x2448 and 310 us for 64 ragged images of 47 Mpx in all, now
// 36 and 217.
constexpr int kCopyRows = 8, kCopyColsBig = 512, kCopyColsSmall = 128, kCopyColsSingle = 32;

struct CopyTile {
  int y, x0, x1;  // the warp's row and its pixels [x0, x1); y < 0: none
};

__device__ __forceinline__ CopyTile copy_tile(const Inst& I, int cols) {
  const int nc = (I.w + cols - 1) / cols;
  const int rb = (int)blockIdx.x / nc, cb = (int)blockIdx.x - rb * nc;
  const int y = rb * kCopyRows + (int)(threadIdx.x >> 5);
  return CopyTile{y < I.h ? y : -1, cb * cols, min((cb + 1) * cols, I.w)};
}

__device__ __forceinline__ bool aligned16(const void* p) {
  return (reinterpret_cast<unsigned long long>(p) & 15ull) == 0;
}

__device__ __forceinline__ void store4(float* d, float4 v) {
  *reinterpret_cast<float4*>(d) = v;
}
__device__ __forceinline__ void store4(__nv_bfloat16* d, float4 v) {
  __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  uint2 u;
  u.x = *reinterpret_cast<unsigned*>(&a);
  u.y = *reinterpret_cast<unsigned*>(&b);
  *reinterpret_cast<uint2*>(d) = u;
}

// One instance's dense images (g null: the guide stays; c null: ones) into
// its pitched planes at `off`.
template <typename TS>
__device__ __forceinline__ void ingest_tile(const Inst& I, const uchar4* g, const float* t,
                                            const float* c, uchar4* __restrict__ guide,
                                            TS* __restrict__ target, TS* __restrict__ conf,
                                            int cs, int cols) {
  const CopyTile T = copy_tile(I, cols);
  if (T.y < 0) return;
  const int lane = threadIdx.x & 31;
  const long long srow = (long long)T.y * I.w, drow = I.off + (long long)T.y * I.pitch;
  if ((I.w & 3) == 0 && aligned16(g) && aligned16(t) && aligned16(c)) {
#pragma unroll
    for (int u = 0; u < kCopyColsBig / 128; ++u) {
      const int x = T.x0 + 4 * lane + 128 * u;
      if (x >= T.x1) break;
      const float4 tv = __ldg(reinterpret_cast<const float4*>(t + srow + x));
      const float4 cv = c ? __ldg(reinterpret_cast<const float4*>(c + srow + x))
                          : make_float4(1.f, 1.f, 1.f, 1.f);
      if (g) {
        uint4 q = __ldg(reinterpret_cast<const uint4*>(g + srow + x));
        if (cs != DTSGB_RGB) {
          unsigned* w = &q.x;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uchar4 r = convert_pixel(*reinterpret_cast<const uchar4*>(w + k), cs);
            w[k] = *reinterpret_cast<const unsigned*>(&r);
          }
        }
        *reinterpret_cast<uint4*>(guide + drow + x) = q;
      }
      store4(target + drow + x, tv);
      store4(conf + drow + x, cv);
    }
    return;
  }
  constexpr int U = 4;  // pixels whose loads are issued before any store
  for (int xb = T.x0 + lane; xb < T.x1; xb += 32 * U) {
    unsigned q[U];
    float tv[U], cv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int x = min(xb + 32 * u, I.w - 1);  // past the row: a copy, not stored
      tv[u] = __ldg(t + srow + x);
      cv[u] = c ? __ldg(c + srow + x) : 1.f;
      q[u] = g ? __ldg(reinterpret_cast<const unsigned*>(g + srow + x)) : 0u;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int x = xb + 32 * u;
      if (x >= T.x1) break;
      if (g) {
        const uchar4 p = *reinterpret_cast<const uchar4*>(q + u);
        guide[drow + x] = cs == DTSGB_RGB ? p : convert_pixel(p, cs);
      }
      target[drow + x] = store_cast<TS>(tv[u]);
      conf[drow + x] = store_cast<TS>(cv[u]);
    }
  }
}

// One instance's dense float image <-> its rows of a pitched plane.
template <bool TO_ARENA>
__device__ __forceinline__ void copy_tile_f32(const Inst& I, float* dense, float* arena,
                                              int cols) {
  const CopyTile T = copy_tile(I, cols);
  if (T.y < 0) return;
  const int lane = threadIdx.x & 31;
  float* d = dense + (long long)T.y * I.w;
  float* a = arena + I.off + (long long)T.y * I.pitch;
  const float* from = TO_ARENA ? d : a;
  float* to = TO_ARENA ? a : d;
  if ((I.w & 3) == 0 && aligned16(dense)) {
#pragma unroll
    for (int u = 0; u < kCopyColsBig / 128; ++u) {
      const int x = T.x0 + 4 * lane + 128 * u;
      if (x >= T.x1) break;
      *reinterpret_cast<float4*>(to + x) = *reinterpret_cast<const float4*>(from + x);
    }
    return;
  }
  constexpr int U = 4;
  for (int xb = T.x0 + lane; xb < T.x1; xb += 32 * U) {
    float v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = from[min(xb + 32 * u, I.w - 1)];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (xb + 32 * u < T.x1) to[xb + 32 * u] = v[u];
  }
}

// Dense staged images -> pitched planes: the guide (color-converted; not
// written when guide is null), target and confidence in the storage type.
template <typename TS>
__global__ void __launch_bounds__(256)
    k_ingest(const Inst* __restrict__ insts, const long long* __restrict__ soff,
             const uchar4* __restrict__ s_rgba, const float* __restrict__ s_t,
             const float* __restrict__ s_c, uchar4* __restrict__ guide,
             TS* __restrict__ target, TS* __restrict__ conf, int cs, int cols) {
  const Inst I = insts[blockIdx.y];
  const long long so = soff[blockIdx.y];
  ingest_tile<TS>(I, guide ? s_rgba + so : nullptr, s_t + so, s_c + so, guide, target, conf, cs,
                  cols);
}

// Dense staged plane -> pitched plane (gradient uploads).  Downloads stay
// row-by-row DMA copies: those need no SM, so in a pipeline they do not wait
// behind another chunk's solve.
__global__ void __launch_bounds__(256)
    k_unstage(const Inst* __restrict__ insts, const long long* __restrict__ soff, float* src,
              float* dst, int cols) {
  copy_tile_f32<true>(insts[blockIdx.y], src + soff[blockIdx.y], dst, cols);
}

// Blocks of the copy kernels (every instance's row blocks times its column
// blocks on x, the instances on y) and their columns: the small ones where
// the big ones would leave the SMs fewer than four blocks each.
dim3 copy_grid(dtsgb_batch_t b, int* cols) {
  auto blocks = [&](int c, long long* most) {
    long long sum = 0;
    *most = 1;
    for (const Inst& I : b->inst) {
      const long long k =
          (long long)((I.h + kCopyRows - 1) / kCopyRows) * ((I.w + c - 1) / c);
      *most = std::max(*most, k);
      sum += k;
    }
    return sum;
  };
  long long most = 1;
  *cols = kCopyColsBig;
  if (blocks(kCopyColsBig, &most) < 4 * 152) {
    bool single = false;
    for (const Inst& I : b->inst) single = single || (I.w & 3) != 0;
    blocks(*cols = single ? kCopyColsSingle : kCopyColsSmall, &most);
  }
  return dim3((unsigned)most, (unsigned)b->n);
}

int ensure_stage(dtsgb_batch_t b) {
  if (b->stage) return DTSGB_OK;
  return dalloc(&b->stage, (size_t)b->dense * 12);
}

// Float region k (0..2) of the staging area.
float* stage_plane(dtsgb_batch_t b, int k) {
  return reinterpret_cast<float*>(b->stage + (size_t)b->dense * 4 * k);
}

// n host images -> pitched device plane, through staging region `region`.
int host_upload_plane(dtsgb_batch_t b, const float* const* src, float* dst, int region) {
  int st = ensure_stage(b);
  if (st) return st;
  float* d = stage_plane(b, region);
  for (int i = 0; i < b->n; ++i) {
    const Inst& I = b->inst[i];
    DTSGB_CUDA(cudaMemcpyAsync(d + b->soff[i], src[i], (size_t)I.w * I.h * 4,
                               cudaMemcpyHostToDevice, b->stream));
  }
  int cols = 0;
  const dim3 grid = copy_grid(b, &cols);
  k_unstage<<<grid, 256, 0, b->stream>>>(b->d_inst, b->d_soff, d, dst, cols);
  DTSGB_CUDA(cudaGetLastError());
  return DTSGB_OK;
}

// Caller pointers of up to kPtrs instances, handed to a kernel by value: a
// table in device memory would cost a copy from pageable host memory, which
// also waits for the stream, before each launch.
constexpr int kPtrs = 128;
struct PtrTable {
  void* p[kPtrs];
};
PtrTable ptr_table(const void* const* ptrs, int first, int n) {
  PtrTable t = {};
  for (int i = 0; ptrs && i < n; ++i) t.p[i] = const_cast<void*>(ptrs[first + i]);
  return t;
}

// Caller device images (dense W x H, one pointer each; null: skipped) <->
// pitched arena plane: one kernel instead of a row-by-row copy per image.
template <bool TO_ARENA>
__global__ void __launch_bounds__(256)
    k_user_copy(const Inst* __restrict__ insts, const __grid_constant__ PtrTable user,
                float* arena, int cols) {
  float* u = static_cast<float*>(user.p[blockIdx.y]);
  if (u) copy_tile_f32<TO_ARENA>(insts[blockIdx.y], u, arena, cols);
}

// Copies between n caller device images and an arena plane.
int user_plane_copy(dtsgb_batch_t b, float* const* user, float* arena, bool to_arena) {
  int cols = 0;
  dim3 grid = copy_grid(b, &cols);
  for (int first = 0; first < b->n; first += kPtrs) {
    grid.y = (unsigned)std::min(kPtrs, b->n - first);
    const PtrTable t = ptr_table(reinterpret_cast<const void* const*>(user), first, (int)grid.y);
    if (to_arena)
      k_user_copy<true><<<grid, 256, 0, b->stream>>>(b->d_inst + first, t, arena, cols);
    else
      k_user_copy<false><<<grid, 256, 0, b->stream>>>(b->d_inst + first, t, arena, cols);
  }
  DTSGB_CUDA(cudaGetLastError());
  return DTSGB_OK;
}

// Caller device images -> pitched planes (the _device uploads): the guide
// (color-converted; not written when guide is null), target and confidence in
// the storage type; a null confidence image stands for ones.
template <typename TS>
__global__ void __launch_bounds__(256)
    k_ingest_ptr(const Inst* __restrict__ insts, const __grid_constant__ PtrTable rgba,
                 const __grid_constant__ PtrTable tgt, const __grid_constant__ PtrTable cnf,
                 uchar4* __restrict__ guide, TS* __restrict__ target, TS* __restrict__ conf,
                 int cs, int cols) {
  const int i = blockIdx.y;
  ingest_tile<TS>(insts[i], static_cast<const uchar4*>(rgba.p[i]),
                  static_cast<const float*>(tgt.p[i]), static_cast<const float*>(cnf.p[i]), guide,
                  target, conf, cs, cols);
}

int device_ingest(dtsgb_batch_t b, int cs, const void* const* rgba,
                  const float* const* target, const float* const* conf) {
  int cols = 0;
  dim3 grid = copy_grid(b, &cols);
  uchar4* g = rgba ? b->guide : nullptr;
  for (int first = 0; first < b->n; first += kPtrs) {
    const int m = std::min(kPtrs, b->n - first);
    grid.y = (unsigned)m;
    const PtrTable tr = ptr_table(rgba, first, m);
    const PtrTable tt = ptr_table(reinterpret_cast<const void* const*>(target), first, m);
    const PtrTable tc = ptr_table(reinterpret_cast<const void* const*>(conf), first, m);
    if (b->st == Storage::F32)
      k_ingest_ptr<float><<<grid, 256, 0, b->stream>>>(b->d_inst + first, tr, tt, tc, g,
                                                       (float*)b->target, (float*)b->conf, cs,
                                                       cols);
    else
      k_ingest_ptr<__nv_bfloat16><<<grid, 256, 0, b->stream>>>(
          b->d_inst + first, tr, tt, tc, g, (__nv_bfloat16*)b->target, (__nv_bfloat16*)b->conf,
          cs, cols);
  }
  DTSGB_CUDA(cudaGetLastError());
  if (rgba) ++b->guide_gen;
  b->dts_res = -1;
  b->grad_n = -1;
  b->hfbs_done = false;
  b->hgrad_ready = false;
  return DTSGB_OK;
}

// Host upload: one contiguous copy per image and plane into the staging
// area (pinned host memory makes them asynchronous), ones for missing
// confidences, then k_ingest.  rgba null: targets only (guides kept).
int host_ingest(dtsgb_batch_t b, int cs, const void* const* rgba,
                const float* const* target, const float* const* conf, bool sync_host) {
  if (int st = ensure_stage(b)) return st;
  uchar4* s_rgba = reinterpret_cast<uchar4*>(b->stage);
  float* s_t = reinterpret_cast<float*>(b->stage + (size_t)b->dense * 4);
  float* s_c = reinterpret_cast<float*>(b->stage + (size_t)b->dense * 8);
  for (int i = 0; i < b->n; ++i) {
    const Inst& I = b->inst[i];
    const size_t px = (size_t)I.w * I.h;
    const long long o = b->soff[i];
    if (rgba)
      DTSGB_CUDA(cudaMemcpyAsync(s_rgba + o, rgba[i], px * 4, cudaMemcpyHostToDevice,
                                 b->stream));
    DTSGB_CUDA(cudaMemcpyAsync(s_t + o, target[i], px * 4, cudaMemcpyHostToDevice,
                               b->stream));
    if (conf && conf[i]) {
      DTSGB_CUDA(cudaMemcpyAsync(s_c + o, conf[i], px * 4, cudaMemcpyHostToDevice,
                                 b->stream));
    } else {
      int st = launch_fill_storage(Storage::F32, s_c + o, (long long)px, 1.f, b->stream);
      if (st) return st;
    }
  }
  int cols = 0;
  const dim3 grid = copy_grid(b, &cols);
  uchar4* g = rgba ? b->guide : nullptr;
  if (b->st == Storage::F32)
    k_ingest<float><<<grid, 256, 0, b->stream>>>(b->d_inst, b->d_soff, s_rgba, s_t, s_c, g,
                                                 (float*)b->target, (float*)b->conf, cs, cols);
  else
    k_ingest<__nv_bfloat16><<<grid, 256, 0, b->stream>>>(
        b->d_inst, b->d_soff, s_rgba, s_t, s_c, g, (__nv_bfloat16*)b->target,
        (__nv_bfloat16*)b->conf, cs, cols);
  DTSGB_CUDA(cudaGetLastError());
  if (rgba) ++b->guide_gen;
  b->dts_res = -1;
  b->grad_n = -1;
  b->hfbs_done = false;
  b->hgrad_ready = false;
  if (sync_host) DTSGB_CUDA(cudaStreamSynchronize(b->stream));
  return DTSGB_OK;
}

// sync_host: a host upload returns only when the copies are done (the
// reference's CopyTo semantics; the host buffers may be reused at once).
int batch_upload_targets(dtsgb_batch_t b, const float* const* target,
                         const float* const* conf, cudaMemcpyKind kind,
                         bool sync_host = true) {
  if (kind == cudaMemcpyHostToDevice)
    return host_ingest(b, DTSGB_RGB, nullptr, target, conf, sync_host);
  return device_ingest(b, DTSGB_RGB, nullptr, target, conf);
}

int batch_upload(dtsgb_batch_t b, int cs, const void* const* rgba,
                 const float* const* target, const float* const* conf,
                 cudaMemcpyKind kind, bool sync_host = true) {
  if (!b || !rgba || !target) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null argument");
  if (cs < DTSGB_RGB || cs > DTSGB_YYY)
    return fail(DTSGB_ERR_INVALID_ARGUMENT, "invalid color space");
  for (int i = 0; i < b->n; ++i)
    if (!rgba[i] || !target[i])
      return fail(DTSGB_ERR_INVALID_ARGUMENT, "null image pointer");
  if (kind == cudaMemcpyHostToDevice)
    return host_ingest(b, cs, rgba, target, conf, sync_host);
  return device_ingest(b, cs, rgba, target, conf);
}

// The HFBS gradient arena for K heavy-ball steps over tv voxels (the choice
// of segment as for the DTS checkpoints: every iterate when that fits in a
// quarter of the free device memory, else about sqrt(K) steps), and the
// three pixel planes of the backward.
int hfbs_prepare_grad(dtsgb_batch_t b, int K, long long tv) {
  int S = b->grad_seg_req;
  if (K <= 1) S = 1;
  if (S <= 0 && b->hgrad_seg == 1 && b->hgcap >= (size_t)(hfbs_grad_planes(K, 1) * tv))
    S = 1;  // every iterate already held: no memory query
  if (S <= 0) {
    size_t fr = 0, tot = 0;
    DTSGB_CUDA(cudaMemGetInfo(&fr, &tot));
    const double avail = (double)fr + (double)b->hgcap * 4.0;
    S = (double)hfbs_grad_planes(K, 1) * tv * 4.0 <= avail / 4
            ? 1
            : std::max(2, (int)std::ceil(std::sqrt((double)K)));
  }
  S = std::min(S, std::max(K, 1));
  const long long need = hfbs_grad_planes(K, S) * tv;
  if ((size_t)need > b->hgcap) {
    DTSGB_CUDA(cudaStreamSynchronize(b->stream));  // a backward may still read it
    dfree(b->hgbuf);
    b->hgcap = 0;
    if (int st = dalloc(&b->hgbuf, (size_t)need)) return st;
    b->hgcap = (size_t)need;
    drop_graph(b, b->g_hbwd);
  }
  if (!b->hpix) {
    if (int st = dalloc(&b->hpix, (size_t)(3 * b->total))) return st;
  }
  hfbs_carve_grad(b->hgs, b->hgbuf, K, S, tv);
  b->hgrad_seg = S;
  b->hgrad_planes = (int)hfbs_grad_planes(K, S);
  return DTSGB_OK;
}

int ensure_hfbs_buffers(dtsgb_batch_t b, long long voxels, long long planes,
                        long long slice_voxels) {
  if (voxels > b->gcap) {
    for (auto& p : b->hg) dfree(p);
    b->gcap = 0;
    b->nkey.gen = ~0ull;  // the normalisation is gone with the old planes
    for (int k = 0; k < HG_NUM; ++k) {
      int st = dalloc(&b->hg[k], (size_t)voxels);
      if (st) return st;
    }
    b->gcap = voxels;
    drop_graph(b, b->g_hfbs);
  }
  if (planes > b->ocap) {
    dfree(b->ovf);
    int st = dalloc(&b->ovf, (size_t)planes);
    if (st) return st;
    b->ocap = planes;
    drop_graph(b, b->g_hfbs);
  }
  if (slice_voxels > b->scap) {
    dfree(b->sgrid);
    int st = dalloc(&b->sgrid, (size_t)slice_voxels);
    if (st) return st;
    b->scap = slice_voxels;
    drop_graph(b, b->g_hfbs);
  }
  return DTSGB_OK;
}

}  // namespace

namespace {
// Mean device time of `reps` runs of `run` on the batch stream (after one
// untimed run, which also captures the graph).
template <typename F>
int time_runs(dtsgb_batch_t b, int reps, F run, float* ms) {
  int st = run();
  if (st) return st;
  cudaEvent_t e0, e1;
  DTSGB_CUDA(cudaEventCreate(&e0));
  cudaError_t e = cudaEventCreate(&e1);
  if (e != cudaSuccess) {
    cudaEventDestroy(e0);
    return cuda_fail(e, "cudaEventCreate");
  }
  e = cudaEventRecord(e0, b->stream);
  for (int r = 0; r < reps && !st && e == cudaSuccess; ++r) st = run();
  if (!st && e == cudaSuccess) e = cudaEventRecord(e1, b->stream);
  if (!st && e == cudaSuccess) e = cudaEventSynchronize(e1);
  float t = 0.f;
  if (!st && e == cudaSuccess) e = cudaEventElapsedTime(&t, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (st) return st;
  if (e != cudaSuccess) return cuda_fail(e, "autotune timing");
  *ms = t / reps;
  return DTSGB_OK;
}
}  // namespace

extern "C" {

DTSGB_API int dtsgb_batch_create(int n, const int* widths, const int* heights,
                                 unsigned flags, dtsgb_batch_t* out) {
  if (!out || !widths || !heights || n <= 0)
    return fail(DTSGB_ERR_INVALID_ARGUMENT, "bad batch description");
  *out = nullptr;
  for (int i = 0; i < n; ++i)
    if (widths[i] <= 0 || heights[i] <= 0)
      return fail(DTSGB_ERR_INVALID_DIMS, "instance dims must be positive");
  dtsgb_batch_t b = new dtsgb_batch_s();
  b->n = n;
  b->flags = flags;
  b->st = (flags & DTSGB_FLAG_BF16_STORAGE) ? Storage::BF16 : Storage::F32;
  b->ref_y = (flags & DTSGB_FLAG_FIX_Y_LIMIT) ? 0 : 1;
  long long off = 0, tiles64 = 0;
  for (int i = 0; i < n; ++i)
    tiles64 += (long long)((widths[i] + kIterTW - 1) / kIterTW) *
               ((heights[i] + kIterTH - 1) / kIterTH);
  b->small = use_small_iter_tiles(tiles64);
  for (int i = 0; i < n; ++i) {
    Inst I{widths[i], heights[i], round_up(widths[i], 32), 0, off};
    b->inst.push_back(I);
    b->soff.push_back(b->dense);
    b->dense += (long long)widths[i] * heights[i];
    off += (long long)I.pitch * I.h;
  }
  b->total = off;
  int st = DTSGB_OK;
  cudaError_t e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    delete b;
    return cuda_fail(e, "cudaStreamCreate");
  }
  b->own_stream = true;
  const size_t T = (size_t)b->total;
  if (!st) st = dalloc(&b->guide, T);
  if (!st) st = dalloc((char**)&b->target, T * b->tsize());
  if (!st) st = dalloc((char**)&b->conf, T * b->tsize());
  if (!st) st = dalloc(&b->bounds, T);
  if (!st) st = dalloc(&b->v[0], T);
  if (!st) st = dalloc(&b->v[1], T);
  if (!st) st = dalloc(&b->hout, T);
  if (!st) st = dalloc(&b->d_inst, (size_t)n);
  if (!st) st = dalloc(&b->d_hinst, (size_t)n);
  if (!st) st = dalloc(&b->d_soff, (size_t)n);
  if (!st && n > 1) {
    // room for four halos' block tables (16 bytes a block of some 1000 pixels)
    for (int halo : {8, 30, 64, 253}) {
      const dim3 t = pass_block_totals(b, halo);
      b->pass_room = std::max(b->pass_room, 4 * ((size_t)t.x + t.y));
    }
    b->pass_mem.push_back(nullptr);
    st = dalloc(&b->pass_mem.back(), b->pass_room);
    b->pass_left = b->pass_room;
  }
  if (!st) {
    e = upload_table(b->d_inst, b->inst.data(), n * sizeof(Inst));
    if (e == cudaSuccess)
      e = upload_table(b->d_soff, b->soff.data(), n * sizeof(long long));
    if (e != cudaSuccess) st = cuda_fail(e, "batch tables");
  }
  if (st) {
    batch_free(b);
    delete b;
    return st;
  }
  *out = b;
  return DTSGB_OK;
}

DTSGB_API int dtsgb_batch_destroy(dtsgb_batch_t b) {
  if (!b) return DTSGB_OK;
  if (b->stream) cudaStreamSynchronize(b->stream);
  batch_free(b);
  delete b;
  return DTSGB_OK;
}

DTSGB_API int dtsgb_batch_set_stream(dtsgb_batch_t b, void* stream) {
  if (!b) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null handle");
  if (!b->own_stream && same_stream(b->stream, stream)) return DTSGB_OK;
  DTSGB_CUDA(cudaStreamSynchronize(b->stream));
  if (b->own_stream) cudaStreamDestroy(b->stream);
  b->own_stream = false;
  b->stream = (cudaStream_t)stream;
  if (!stream) {
    DTSGB_CUDA(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
    b->own_stream = true;
  }
  return DTSGB_OK;
}

DTSGB_API int dtsgb_batch_use_graphs(dtsgb_batch_t b, int enable) {
  if (!b) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null handle");
  b->use_graphs = enable != 0;
  if (!b->use_graphs) {
    drop_graph(b, b->g_dts);
    drop_graph(b, b->g_hfbs);
  }
  return DTSGB_OK;
}

DTSGB_API int dtsgb_batch_upload(dtsgb_batch_t b, int cs, const void* const* rgba,
                                 const float* const* target,
                                 const float* const* conf) {
  return batch_upload(b, cs, rgba, target, conf, cudaMemcpyHostToDevice);
}

DTSGB_API int dtsgb_batch_upload_targets(dtsgb_batch_t b, const float* const* target,
                                         const float* const* conf) {
  if (!b || !target) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null argument");
  for (int i = 0; i < b->n; ++i)
    if (!target[i]) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null image pointer");
  return batch_upload_targets(b, target, conf, cudaMemcpyHostToDevice);
}

DTSGB_API int dtsgb_batch_upload_targets_device(dtsgb_batch_t b,
                                                const float* const* target,
                                                const float* const* conf) {
  if (!b || !target) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null argument");
  for (int i = 0; i < b->n; ++i)
    if (!target[i]) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null image pointer");
  return batch_upload_targets(b, target, conf, cudaMemcpyDeviceToDevice);
}

DTSGB_API int dtsgb_batch_upload_device(dtsgb_batch_t b, int cs,
                                        const void* const* rgba,
                                        const float* const* target,
                                        const float* const* conf) {
  return batch_upload(b, cs, rgba, target, conf, cudaMemcpyDeviceToDevice);
}

DTSGB_API int dtsgb_batch_solve_dts(dtsgb_batch_t b, const dtsgb_filter_params* f,
                                    const dtsgb_optimize_params* p,
                                    float overwrite) {
  if (!b || !f || !p) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null argument");
  if (!finite_pos(f->sigma_x) || !finite_pos(f->sigma_y) || !finite_pos(f->sigma_r))
    return fail(DTSGB_ERR_INVALID_ARGUMENT, "filter sigmas must be finite, positive");
  if (p->loss < DTSGB_L1 || p->loss > DTSGB_CHARBONNIER)
    return fail(DTSGB_ERR_INVALID_ARGUMENT, "invalid loss");
  if (p->num_iterations < 0)
    return fail(DTSGB_ERR_INVALID_ARGUMENT, "num_iterations < 0");
  if (!finite_pos(p->sigma_z) || p->sigma_z >= 254.f)
    return fail(DTSGB_ERR_UNSUPPORTED, "sigma_z must be in (0, 254)");
  const float rx = f->sigma_x / f->sigma_r, ry = f->sigma_y / f->sigma_r;
  const int halo = (int)std::floor(p->sigma_z);
  const bool iterate = p->loss != DTSGB_L1 && p->num_iterations > 0;
  bool fresh = false;
  if (iterate)
    if (int st = ensure_pass_blocks(b, halo, &fresh)) return st;
  const DtsLaunch Li = iter_launch(b, halo);
  const bool over = overwrite > 0.f && overwrite < 1.f;
  const int n_kept = iterate ? p->num_iterations : 0;
  b->grad_n = -1;
  if (b->grad) {
    if (iterate && over)
      return fail(DTSGB_ERR_UNSUPPORTED,
                  "gradients are not available with the confidence overwrite");
    int seg = b->grad_seg_req;
    if (seg <= 0) {
      // automatic: every iterate kept (nothing recomputed by the backward)
      // when its N + 4 planes fit in a quarter of the free device memory (or
      // are held already), else the fewest planes
      const int n = std::max(n_kept, 1);
      const size_t need = (size_t)(n + 4) * (size_t)b->total * sizeof(float);
      size_t free_b = 0, total_b = 0;
      const bool held = b->grad_seg == 1 && b->gplanes.size() == (size_t)n + 4;
      if (!held) DTSGB_CUDA(cudaMemGetInfo(&free_b, &total_b));
      seg = held || need <= free_b / 4 ? 1 : dts_checkpoint_segment(n);
    }
    int st = ensure_grad_planes(b, n_kept, seg);
    if (st) return st;
  }
  const dtsgb_batch_s::BoundsKey bk{b->guide_gen, rx, ry, p->sigma_z, b->ref_y};
  // (the passes are dependent launches that read their block before they wait:
  // with new tables the bounds pass, a plain launch, comes in between)
  const bool keep_bounds = b->reuse && !fresh && std::memcmp(&bk, &b->bkey, sizeof bk) == 0;
  auto bounds = [&]() -> int {
    if (keep_bounds) return DTSGB_OK;  // same guide and sigmas: windows unchanged
    return launch_bounds(Li, b->guide, b->bounds, rx, ry, p->sigma_z, p->sigma_z,
                         b->ref_y, b->stream);
  };
  auto enqueue = [&]() -> int {
    if (b->grad && iterate) {
      const IterMode mode = p->loss == DTSGB_L2 ? IterMode::L2 : IterMode::CHARB;
      int st = bounds();
      if (st) return st;
      return dts_forward_checkpointed(Li, b->st, mode, grad_view(b, n_kept), b->target,
                                      b->conf, b->bounds, p->lambda, p->step_size, halo,
                                      p->num_iterations, b->v[0], b->v[1], b->stream);
    }
    if (!iterate) return launch_init_var(Li, b->st, b->target, b->v[0], b->stream);
    const float* cur = nullptr;
    int st = first_iterate(Li, b->st, b->target, b->v[0], &cur, b->stream);
    if (st) return st;
    st = bounds();
    if (st) return st;
    const IterMode mode = p->loss == DTSGB_L2 ? IterMode::L2 : IterMode::CHARB;
    for (int it = 0; it < p->num_iterations; ++it) {
      st = launch_dts_iter(Li, b->st, mode, cur, b->v[1], b->v[0], b->target, b->conf, b->bounds,
                           p->lambda, p->step_size, overwrite, it + 1 < p->num_iterations, halo,
                           b->stream);
      if (st) return st;
      cur = b->v[0];
    }
    return DTSGB_OK;
  };
  std::vector<char> key;
  key_append(key, *f);
  key_append(key, *p);
  key_append(key, overwrite);
  key_append(key, b->grad);
  key_append(key, b->grad_seg);
  key_append(key, keep_bounds);
  int st = run_graph(b, b->g_dts, key, enqueue);
  if (st) {
    b->bkey.gen = ~0ull;
    return st;
  }
  if (iterate) b->bkey = bk;
  if (iterate && !keep_bounds && callers_capture(b)) b->bkey.gen = ~0ull;  // not run yet
  b->dts_res = 0;
  if (b->grad) {
    b->grad_n = n_kept;
    b->gopt = *p;
    b->ghalo = (float)halo;
  }
  return DTSGB_OK;
}

DTSGB_API int dtsgb_batch_enable_grad(dtsgb_batch_t b, int enable, int segment) {
  if (!b) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null handle");
  if (segment < 0) return fail(DTSGB_ERR_INVALID_ARGUMENT, "segment < 0");
  if (b->grad != (enable != 0) || b->grad_seg_req != segment) {
    DTSGB_CUDA(cudaStreamSynchronize(b->stream));
    drop_graph(b, b->g_dts);
    drop_graph(b, b->g_bwd);
    drop_graph(b, b->g_hfbs);
    drop_graph(b, b->g_hbwd);
  }
  b->grad = enable != 0;
  b->grad_seg_req = segment;
  b->grad_n = -1;
  b->hgrad_ready = false;
  if (!b->grad) {
    free_grad_planes(b);
    dfree(b->hgbuf);
    dfree(b->hpix);
    b->hgcap = 0;
    b->hgrad_seg = b->hgrad_planes = 0;
  }
  return DTSGB_OK;
}

DTSGB_API int dtsgb_batch_grad_info(dtsgb_batch_t b, int* segment, int* planes) {
  if (!b || !segment || !planes) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null argument");
  *segment = b->grad_n >= 0 ? b->grad_seg : 0;
  *planes = (int)b->gplanes.size();
  return DTSGB_OK;
}

static int batch_backward(dtsgb_batch_t b, const float* const* grad_out,
                          float* const* grad_t, float* const* grad_c,
                          cudaMemcpyKind up, cudaMemcpyKind down, bool sync_host = true) {
  if (!b || !grad_out) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null argument");
  if (b->grad_n < 0)
    return fail(DTSGB_ERR_INVALID_ARGUMENT,
                "no DTS solve with gradients enabled since the last upload");
  for (int i = 0; i < b->n; ++i)
    if (!grad_out[i]) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null gradient pointer");
  const int n_iter = b->grad_n;
  DtsGrad G = grad_view(b, n_iter);
  if (up == cudaMemcpyHostToDevice) {
    if (int st = host_upload_plane(b, grad_out, G.g[0], 0)) return st;
  } else {
    if (int st = user_plane_copy(b, const_cast<float* const*>(grad_out), G.g[0], true))
      return st;
  }
  const dtsgb_optimize_params p = b->gopt;
  const int halo = (int)b->ghalo;
  const DtsLaunch Li = iter_launch(b, halo);
  auto enqueue = [&]() -> int {
    const IterMode mode = p.loss == DTSGB_L2 ? IterMode::L2 : IterMode::CHARB;
    return dts_backward(Li, b->d_inst, b->n, b->total, b->st, mode, G, b->target, b->conf,
                        b->bounds, p.lambda, p.step_size, halo, n_iter, b->v[1],
                        grad_plane_t(b), grad_plane_c(b), b->stream);
  };
  std::vector<char> key;
  key_append(key, p);
  key_append(key, n_iter);
  key_append(key, b->grad_seg);
  int st = run_graph(b, b->g_bwd, key, enqueue);
  if (st) return st;
  for (int k = 0; k < 2; ++k) {
    float* const* dst = k == 0 ? grad_t : grad_c;
    const float* src = k == 0 ? grad_plane_t(b) : grad_plane_c(b);
    if (!dst) continue;
    if (down == cudaMemcpyDeviceToDevice) {
      if (int st = user_plane_copy(b, dst, const_cast<float*>(src), false)) return st;
      continue;
    }
    for (int i = 0; i < b->n; ++i) {
      if (!dst[i]) continue;
      const Inst& I = b->inst[i];
      const size_t wb = (size_t)I.w * 4;
      DTSGB_CUDA(cudaMemcpy2DAsync(dst[i], wb, src + I.off, (size_t)I.pitch * 4, wb, I.h,
                                   down, b->stream));
    }
  }
  if (down == cudaMemcpyDeviceToHost && sync_host)
    DTSGB_CUDA(cudaStreamSynchronize(b->stream));
  return DTSGB_OK;
}

DTSGB_API int dtsgb_batch_dts_backward(dtsgb_batch_t b, const float* const* grad_out,
                                       float* const* grad_target,
                                       float* const* grad_confidence) {
  return batch_backward(b, grad_out, grad_target, grad_confidence, cudaMemcpyHostToDevice,
                        cudaMemcpyDeviceToHost);
}

DTSGB_API int dtsgb_batch_dts_backward_device(dtsgb_batch_t b,
                                              const float* const* grad_out,
                                              float* const* grad_target,
                                              float* const* grad_confidence) {
  return batch_backward(b, grad_out, grad_target, grad_confidence,
                        cudaMemcpyDeviceToDevice, cudaMemcpyDeviceToDevice);
}

DTSGB_API int dtsgb_batch_solve_hfbs(dtsgb_batch_t b, const dtsgb_hfbs_params* p) {
  if (!b || !p) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null argument");
  if (!finite_pos(p->sigma_x) || !finite_pos(p->sigma_y) || !finite_pos(p->sigma_l))
    return fail(DTSGB_ERR_INVALID_ARGUMENT, "grid sigmas must be finite, positive");
  if (p->bistoch_iter_max < 0 || p->optim_iter_max < 0)
    return fail(DTSGB_ERR_INVALID_ARGUMENT, "iteration counts must be >= 0");
  const int gl = (int)std::ceil(255.0 / (double)p->sigma_l);
  if (gl > 256) return fail(DTSGB_ERR_UNSUPPORTED, "more than 256 luma bins");
  std::vector<HInst> hi(b->n);
  long long goff = 0, poff = 0, soff = 0, max_vox = 0, max_px = 0, max_cells = 0,
            max_lines = 0;
  for (int i = 0; i < b->n; ++i) {
    const Inst& I = b->inst[i];
    HInst& H = hi[i];
    H.w = I.w;
    H.h = I.h;
    H.pitch = I.pitch;
    H.gx = (int)std::ceil((float)I.w / p->sigma_x);
    H.gy = (int)std::ceil((float)I.h / p->sigma_y);
    H.gl = gl;
    H.px = round_up(H.gx, 4);
    H.cov_x = H.gx % 8 != 0;
    H.cov_y = H.gy % 8 != 0;
    H.cov_l = H.gl % 8 != 0;
    H.ovf_stored = 1;
    H.pix_off = I.off;
    H.grid_off = goff;
    H.plane_off = poff;
    H.slice_off = soff;
    soff += round_up_ll((long long)(H.gx + 1) * (H.gy + 1) * (H.gl + 2), 32);
    const long long vox = (long long)H.gx * H.gy * H.gl;
    goff += round_up_ll((long long)H.px * H.gy * H.gl, 32);
    poff += round_up_ll((long long)H.gx * H.gy, 32);
    max_vox = std::max(max_vox, vox);
    max_px = std::max(max_px, (long long)I.w * I.h);
    max_cells = std::max(max_cells, (long long)H.gx * H.gy);
    max_lines = std::max({max_lines, (long long)H.gy * H.gl, (long long)H.gx * H.gl,
                          (long long)H.gx * H.gy});
  }
  int st = ensure_hfbs_buffers(b, goff, poff, soff);
  if (st) return st;
  const bool same_tables =
      b->hinst.size() == hi.size() &&
      std::memcmp(b->hinst.data(), hi.data(), hi.size() * sizeof(HInst)) == 0;
  if (!same_tables) {
    b->htma.clear();
    b->hinst = hi;
    DTSGB_CUDA(cudaMemcpyAsync(b->d_hinst, b->hinst.data(), hi.size() * sizeof(HInst),
                               cudaMemcpyHostToDevice, b->stream));
    DTSGB_CUDA(cudaStreamSynchronize(b->stream));
  }
  HfbsBatch B{};
  B.d_inst = b->d_hinst;
  B.n_inst = b->n;
  B.max_voxels = max_vox;
  B.total_voxels = goff;
  B.max_pixels = max_px;
  B.max_cells = max_cells;
  B.max_lines = max_lines;
  B.max_rows = 0;
  for (const HInst& H : hi) B.max_rows = std::max(B.max_rows, (long long)H.gy * H.gl);
  B.max_gl = gl;
  B.guide = b->guide;
  B.target = b->target;
  B.conf = b->conf;
  B.st = b->st;
  B.out = b->hout;
  B.count = b->hg[HG_COUNT];
  B.csum = b->hg[HG_CSUM];
  B.b = b->hg[HG_B];
  B.n0 = b->hg[HG_N0];
  B.n1 = b->hg[HG_N1];
  B.invA = b->hg[HG_INVA];
  B.z0 = b->hg[HG_Z0];
  B.z1 = b->hg[HG_Z1];
  B.h = b->hg[HG_H];
  B.t0 = b->hg[HG_T0];
  B.t1 = b->hg[HG_T1];
  B.t2 = b->hg[HG_T2];
  B.sgrid = b->sgrid;
  B.ovf = b->ovf;
  B.keep_debug = false;
  B.h_inst = b->hinst.data();
  B.group_voxels = b->hfbs_group_voxels;
  B.solve_steps = b->hfbs_solve_steps;
  B.tma = &b->htma;
  // the bistochastized normalisation depends only on the guide's bins
  const dtsgb_batch_s::NormKey nk{b->guide_gen, p->sigma_x, p->sigma_y, p->sigma_l,
                                  p->bistoch_iter_max};
  B.reuse_norm = b->reuse && same_tables && std::memcmp(&nk, &b->nkey, sizeof nk) == 0;
  HParams hp{p->sigma_x, p->sigma_y, p->sigma_l, p->lambda, p->alpha, p->beta,
             p->bistoch_iter_max, p->optim_iter_max, p->neg_exp_beta};
  b->hgrad_ready = false;
  if (b->grad) {
    if ((st = hfbs_prepare_grad(b, p->optim_iter_max, goff))) return st;
    B.grad = &b->hgs;
  }
  hfbs_prepare_tma(B, hp, b->stream);  // before any capture of the solve
  std::vector<char> key;
  key_append(key, hp);
  key_append(key, b->hfbs_group_voxels);
  key_append(key, b->hfbs_solve_steps);
  key_append(key, B.reuse_norm);
  key_append(key, b->grad ? b->hgbuf : nullptr);  // the kept iterates' arena
  key_append(key, b->grad ? b->hgrad_seg : 0);
  st = run_graph(b, b->g_hfbs, key, [&]() { return hfbs_enqueue_solve(B, hp, b->stream); });
  if (st) {
    b->nkey.gen = ~0ull;
    return st;
  }
  b->nkey = nk;
  if (!B.reuse_norm && callers_capture(b)) b->nkey.gen = ~0ull;  // not run yet
  b->hfbs_done = true;
  if (b->grad) {
    b->hB = B;
    b->hhp = hp;
    b->hgrad_ready = true;
  }
  return DTSGB_OK;
}

// Adjoint of the last differentiable dtsgb_batch_solve_hfbs (the HFBS
// counterpart of batch_backward): upstream gradients in, dL/dtarget and
// dL/dconfidence out, the launch sequence replayed from a CUDA graph.
static int batch_hfbs_backward(dtsgb_batch_t b, const float* const* grad_out,
                               float* const* grad_t, float* const* grad_c,
                               cudaMemcpyKind up, cudaMemcpyKind down) {
  if (!b || !grad_out) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null argument");
  if (!b->hgrad_ready)
    return fail(DTSGB_ERR_INVALID_ARGUMENT,
                "no HFBS solve with gradients enabled since the last upload");
  for (int i = 0; i < b->n; ++i)
    if (!grad_out[i]) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null gradient pointer");
  float* gout = b->hpix;
  float* gt = b->hpix + b->total;
  float* gc = b->hpix + 2 * b->total;
  if (up == cudaMemcpyHostToDevice) {
    if (int st = host_upload_plane(b, grad_out, gout, 0)) return st;
  } else {
    if (int st = user_plane_copy(b, const_cast<float* const*>(grad_out), gout, true))
      return st;
  }
  std::vector<char> key;
  key_append(key, b->hhp);
  key_append(key, b->hgbuf);
  key_append(key, b->hgrad_seg);
  key_append(key, b->hB.total_voxels);
  int st = run_graph(b, b->g_hbwd, key,
                     [&]() { return hfbs_enqueue_backward(b->hB, b->hhp, gout, gt, gc, b->stream); });
  if (st) return st;
  for (int k = 0; k < 2; ++k) {
    float* const* dst = k == 0 ? grad_t : grad_c;
    const float* src = k == 0 ? gt : gc;
    if (!dst) continue;
    if (down == cudaMemcpyDeviceToDevice) {
      if (int st = user_plane_copy(b, dst, const_cast<float*>(src), false)) return st;
      continue;
    }
    for (int i = 0; i < b->n; ++i) {
      if (!dst[i]) continue;
      const Inst& I = b->inst[i];
      const size_t wb = (size_t)I.w * 4;
      DTSGB_CUDA(cudaMemcpy2DAsync(dst[i], wb, src + I.off, (size_t)I.pitch * 4, wb, I.h,
                                   down, b->stream));
    }
  }
  if (down == cudaMemcpyDeviceToHost) DTSGB_CUDA(cudaStreamSynchronize(b->stream));
  return DTSGB_OK;
}

DTSGB_API int dtsgb_batch_hfbs_backward(dtsgb_batch_t b, const float* const* grad_out,
                                        float* const* grad_target,
                                        float* const* grad_confidence) {
  return batch_hfbs_backward(b, grad_out, grad_target, grad_confidence,
                             cudaMemcpyHostToDevice, cudaMemcpyDeviceToHost);
}

DTSGB_API int dtsgb_batch_hfbs_backward_device(dtsgb_batch_t b, const float* const* grad_out,
                                               float* const* grad_target,
                                               float* const* grad_confidence) {
  return batch_hfbs_backward(b, grad_out, grad_target, grad_confidence,
                             cudaMemcpyDeviceToDevice, cudaMemcpyDeviceToDevice);
}

DTSGB_API int dtsgb_batch_hfbs_grad_info(dtsgb_batch_t b, int* segment, int* planes) {
  if (!b || !segment || !planes) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null argument");
  *segment = b->hgrad_ready ? b->hgrad_seg : 0;
  *planes = b->hgrad_ready ? b->hgrad_planes : 0;
  return DTSGB_OK;
}

DTSGB_API int dtsgb_batch_set_tuning(dtsgb_batch_t b, int knob, long long value) {
  if (!b) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null handle");
  if (knob == DTSGB_TUNE_DTS_TILE) {
    if (value != kIterTW && value != kIterSmallTW)
      return fail(DTSGB_ERR_INVALID_ARGUMENT, "DTS tile must be 64 or 32");
    b->small = value == kIterSmallTW;  // (no solve depends on it)
    return DTSGB_OK;
  }
  if (knob == DTSGB_TUNE_HFBS_GROUP_VOXELS) {
    if (value < 0) return fail(DTSGB_ERR_INVALID_ARGUMENT, "group budget < 0");
    b->hfbs_group_voxels = value;
    return DTSGB_OK;
  }
  if (knob == DTSGB_TUNE_REUSE_GUIDE_STATE) {
    b->reuse = value != 0;
    return DTSGB_OK;
  }
  if (knob == DTSGB_TUNE_BOUNDS_SEGMENT) {
    if (value != 4 && value != 8 && value != 16)
      return fail(DTSGB_ERR_INVALID_ARGUMENT, "bounds segment must be 4, 8 or 16");
    b->bounds_seg = (int)value;
    return DTSGB_OK;
  }
  if (knob == DTSGB_TUNE_HFBS_SOLVE_STEPS) {
    if (value != 1 && value != kHfbsMarchSteps)
      return fail(DTSGB_ERR_INVALID_ARGUMENT, "HFBS steps per launch must be 1 or 4");
    if (value != b->hfbs_solve_steps) b->hgrad_ready = false;  // kept iterates' arithmetic
    b->hfbs_solve_steps = (int)value;
    return DTSGB_OK;
  }
  return fail(DTSGB_ERR_INVALID_ARGUMENT, "unknown tuning knob");
}

DTSGB_API int dtsgb_batch_get_tuning(dtsgb_batch_t b, int knob, long long* value) {
  if (!b || !value) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null argument");
  if (knob == DTSGB_TUNE_DTS_TILE) {
    *value = b->small ? kIterSmallTW : kIterTW;
    return DTSGB_OK;
  }
  if (knob == DTSGB_TUNE_HFBS_GROUP_VOXELS) {
    *value = b->hfbs_group_voxels;
    return DTSGB_OK;
  }
  if (knob == DTSGB_TUNE_REUSE_GUIDE_STATE) {
    *value = b->reuse ? 1 : 0;
    return DTSGB_OK;
  }
  if (knob == DTSGB_TUNE_HFBS_SOLVE_STEPS) {
    *value = b->hfbs_solve_steps;
    return DTSGB_OK;
  }
  if (knob == DTSGB_TUNE_BOUNDS_SEGMENT) {
    *value = b->bounds_seg;
    return DTSGB_OK;
  }
  return fail(DTSGB_ERR_INVALID_ARGUMENT, "unknown tuning knob");
}

DTSGB_API int dtsgb_batch_autotune(dtsgb_batch_t b, const dtsgb_filter_params* f,
                                   const dtsgb_optimize_params* p, float overwrite,
                                   const dtsgb_hfbs_params* hp, int reps) {
  if (!b) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null handle");
  if ((f == nullptr) != (p == nullptr))
    return fail(DTSGB_ERR_INVALID_ARGUMENT, "filter and optimize params go together");
  if (reps < 1) reps = 3;
  // every timed solve does all of its work (no guide state kept across runs)
  const bool reuse = b->reuse;
  b->reuse = false;
  int st = DTSGB_OK;
  // (no knob changes how a DTS solve runs)
  if (hp) {
    auto hfbs = [&]() { return dtsgb_batch_solve_hfbs(b, hp); };
    float best = 3.4e38f;
    long long best_s = kHfbsMarchSteps, best_g = 0;
    for (long long steps : {(long long)kHfbsMarchSteps, 1LL}) {
      if ((st = dtsgb_batch_set_tuning(b, DTSGB_TUNE_HFBS_SOLVE_STEPS, steps))) break;
      for (long long g : {0LL, 1000000LL, 2000000LL, 4000000LL, 8000000LL}) {
        if ((st = dtsgb_batch_set_tuning(b, DTSGB_TUNE_HFBS_GROUP_VOXELS, g))) break;
        float ms = 0.f;
        if ((st = time_runs(b, reps, hfbs, &ms))) break;
        if (ms < best) {
          best = ms;
          best_s = steps;
          best_g = g;
        }
      }
      if (st) break;
    }
    if (!st) st = dtsgb_batch_set_tuning(b, DTSGB_TUNE_HFBS_SOLVE_STEPS, best_s);
    if (!st) st = dtsgb_batch_set_tuning(b, DTSGB_TUNE_HFBS_GROUP_VOXELS, best_g);
  }
  b->reuse = reuse;
  if (st) return st;
  // leave the results of one solve with the chosen setting
  if (f && (st = dtsgb_batch_solve_dts(b, f, p, overwrite))) return st;
  if (hp && (st = dtsgb_batch_solve_hfbs(b, hp))) return st;
  return DTSGB_OK;
}

}  // extern "C"

namespace {

// FNV-1a over bytes: the autotune cache key.
struct Fnv {
  unsigned long long h = 1469598103934665603ull;
  template <typename T>
  void add(const T& v) {
    const unsigned char* q = reinterpret_cast<const unsigned char*>(&v);
    for (size_t i = 0; i < sizeof(T); ++i) h = (h ^ q[i]) * 1099511628211ull;
  }
};

const int kCachedKnobs[4] = {DTSGB_TUNE_DTS_TILE, DTSGB_TUNE_BOUNDS_SEGMENT,
                             DTSGB_TUNE_HFBS_SOLVE_STEPS, DTSGB_TUNE_HFBS_GROUP_VOXELS};

}  // namespace

extern "C" {

DTSGB_API int dtsgb_batch_autotune_cached(dtsgb_batch_t b, const dtsgb_filter_params* f,
                                          const dtsgb_optimize_params* p, float overwrite,
                                          const dtsgb_hfbs_params* hp, int reps,
                                          const char* cache_path, int* from_cache) {
  if (!b || !cache_path) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null argument");
  if ((f == nullptr) != (p == nullptr))
    return fail(DTSGB_ERR_INVALID_ARGUMENT, "filter and optimize params go together");
  int dev = 0;
  DTSGB_CUDA(cudaGetDevice(&dev));
  cudaDeviceProp prop{};
  DTSGB_CUDA(cudaGetDeviceProperties(&prop, dev));
  // key: the device, the batch's shapes and storage, and the parameters
  Fnv k;
  for (const char* c = prop.name; *c; ++c) k.add(*c);
  k.add(prop.multiProcessorCount);
  k.add(b->n);
  k.add(b->flags);
  for (const Inst& I : b->inst) {
    k.add(I.w);
    k.add(I.h);
  }
  k.add(f != nullptr);
  if (f) {
    k.add(*f);
    k.add(*p);
    k.add(overwrite);
  }
  k.add(hp != nullptr);
  if (hp) k.add(*hp);
  char key[32];
  std::snprintf(key, sizeof key, "%016llx", k.h);
  if (from_cache) *from_cache = 0;
  {
    std::ifstream in(cache_path);
    std::string line;
    while (in && std::getline(in, line)) {
      std::istringstream ls(line);
      std::string lk;
      long long v[4];
      if (!(ls >> lk >> v[0] >> v[1] >> v[2] >> v[3]) || lk != key) continue;
      int st = DTSGB_OK;
      for (int i = 0; i < 4 && !st; ++i) st = dtsgb_batch_set_tuning(b, kCachedKnobs[i], v[i]);
      if (st) break;  // a stale line: tune again
      if (f && (st = dtsgb_batch_solve_dts(b, f, p, overwrite))) return st;
      if (hp && (st = dtsgb_batch_solve_hfbs(b, hp))) return st;
      if (from_cache) *from_cache = 1;
      return DTSGB_OK;
    }
  }
  int st = dtsgb_batch_autotune(b, f, p, overwrite, hp, reps);
  if (st) return st;
  std::ofstream out(cache_path, std::ios::app);
  if (out) {
    out << key;
    for (int kn : kCachedKnobs) {
      long long v = 0;
      dtsgb_batch_get_tuning(b, kn, &v);
      out << ' ' << v;
    }
    out << ' ' << prop.name << '\n';
  }
  return DTSGB_OK;  // a cache that cannot be written only costs the next caller a tuning
}

static int batch_download(dtsgb_batch_t b, int which, float* const* dst,
                          cudaMemcpyKind kind, bool sync_host = true) {
  if (!b || !dst) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null argument");
  const float* src = nullptr;
  if (which == 0) {
    if (b->dts_res < 0) return fail(DTSGB_ERR_INVALID_ARGUMENT, "no DTS solve yet");
    src = b->v[b->dts_res];
  } else if (which == 1) {
    if (!b->hfbs_done) return fail(DTSGB_ERR_INVALID_ARGUMENT, "no HFBS solve yet");
    src = b->hout;
  } else {
    return fail(DTSGB_ERR_INVALID_ARGUMENT, "which must be 0 (DTS) or 1 (HFBS)");
  }
  for (int i = 0; i < b->n; ++i)
    if (!dst[i]) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null output pointer");
  if (kind == cudaMemcpyDeviceToDevice)
    return user_plane_copy(b, dst, const_cast<float*>(src), false);
  for (int i = 0; i < b->n; ++i) {
    const Inst& I = b->inst[i];
    const size_t wb = (size_t)I.w * 4;
    DTSGB_CUDA(cudaMemcpy2DAsync(dst[i], wb, src + I.off, (size_t)I.pitch * 4, wb, I.h,
                                 kind, b->stream));
  }
  if (kind == cudaMemcpyDeviceToHost && sync_host)
    DTSGB_CUDA(cudaStreamSynchronize(b->stream));
  return DTSGB_OK;
}

DTSGB_API int dtsgb_batch_download(dtsgb_batch_t b, int which, float* const* dst) {
  return batch_download(b, which, dst, cudaMemcpyDeviceToHost);
}

DTSGB_API int dtsgb_batch_download_device(dtsgb_batch_t b, int which,
                                          float* const* dst) {
  return batch_download(b, which, dst, cudaMemcpyDeviceToDevice);
}

DTSGB_API int dtsgb_batch_debug_plane(dtsgb_batch_t b, int i, int which, void* dst,
                                      long long dst_bytes) {
  if (!b || !dst) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null argument");
  if (i < 0 || i >= b->n) return fail(DTSGB_ERR_INVALID_ARGUMENT, "instance index");
  if (which == DTSGB_BATCH_PLANE_BOUNDS) {
    if (b->dts_res < 0) return fail(DTSGB_ERR_INVALID_ARGUMENT, "no DTS solve yet");
    const Inst& I = b->inst[i];
    const size_t wb = (size_t)I.w * 4;
    if (dst_bytes < (long long)wb * I.h)
      return fail(DTSGB_ERR_INVALID_ARGUMENT, "dst_bytes smaller than W*H*4");
    DTSGB_CUDA(cudaMemcpy2DAsync(dst, wb, b->bounds + I.off, (size_t)I.pitch * 4, wb, I.h,
                                 cudaMemcpyDeviceToHost, b->stream));
  } else if (which >= DTSGB_BATCH_PLANE_COUNT && which <= DTSGB_BATCH_PLANE_B) {
    if (!b->hfbs_done || (int)b->hinst.size() != b->n)
      return fail(DTSGB_ERR_INVALID_ARGUMENT, "no HFBS solve yet");
    const HInst& H = b->hinst[i];
    const long long n = (long long)H.gx * H.gy * H.gl;
    if (dst_bytes < n * 4)
      return fail(DTSGB_ERR_INVALID_ARGUMENT, "dst_bytes smaller than gx*gy*gl*4");
    const int g = which == DTSGB_BATCH_PLANE_COUNT ? HG_COUNT
                  : which == DTSGB_BATCH_PLANE_CSUM ? HG_CSUM : HG_B;
    // rows of px voxels on the device, of gx in dst
    DTSGB_CUDA(cudaMemcpy2DAsync(dst, (size_t)H.gx * 4, b->hg[g] + H.grid_off,
                                 (size_t)H.px * 4, (size_t)H.gx * 4, (size_t)H.gy * H.gl,
                                 cudaMemcpyDeviceToHost, b->stream));
  } else {
    return fail(DTSGB_ERR_INVALID_ARGUMENT, "which must be a DTSGB_BATCH_PLANE_* value");
  }
  DTSGB_CUDA(cudaStreamSynchronize(b->stream));
  return DTSGB_OK;
}


// ---------------------------------------------------------------------------
// Overlapped host-to-host solves: chunks of the instances, each a batch on
// its own stream; every chunk's upload, solves and downloads are enqueued
// without waiting, so copies of one chunk overlap the solves of another.
// ---------------------------------------------------------------------------
struct dtsgb_pipeline_s {
  std::vector<dtsgb_batch_t> chunk;
  std::vector<int> first;  // index of each chunk's first instance
  int n = 0;
};

DTSGB_API int dtsgb_pipeline_destroy(dtsgb_pipeline_t p) {
  if (!p) return DTSGB_OK;
  for (dtsgb_batch_t b : p->chunk) dtsgb_batch_destroy(b);
  delete p;
  return DTSGB_OK;
}

DTSGB_API int dtsgb_pipeline_create(int n, const int* widths, const int* heights,
                                    unsigned flags, int n_chunks, dtsgb_pipeline_t* out) {
  if (!out || !widths || !heights || n <= 0 || n_chunks <= 0)
    return fail(DTSGB_ERR_INVALID_ARGUMENT, "bad pipeline description");
  *out = nullptr;
  long long total = 0;
  for (int i = 0; i < n; ++i) {
    if (widths[i] <= 0 || heights[i] <= 0)
      return fail(DTSGB_ERR_INVALID_DIMS, "instance dims must be positive");
    total += (long long)widths[i] * heights[i];
  }
  n_chunks = std::min(n_chunks, n);
  dtsgb_pipeline_t p = new dtsgb_pipeline_s();
  p->n = n;
  // contiguous runs of instances, cut where the running pixel count passes
  // k / n_chunks of the total
  long long acc = 0;
  int start = 0;
  for (int i = 0; i < n; ++i) {
    acc += (long long)widths[i] * heights[i];
    const int k = (int)p->first.size() + 1;  // chunk being filled, 1-based
    const bool last = i == n - 1;
    const bool cut = acc * n_chunks >= total * k && n - (i + 1) >= n_chunks - k;
    const bool must = n - (i + 1) == n_chunks - k;  // one instance per chunk left
    if (last || ((cut || must) && k < n_chunks)) {
      dtsgb_batch_t b = nullptr;
      int st = dtsgb_batch_create(i + 1 - start, widths + start, heights + start, flags, &b);
      if (st) {
        dtsgb_pipeline_destroy(p);
        return st;
      }
      p->chunk.push_back(b);
      p->first.push_back(start);
      start = i + 1;
    }
  }
  *out = p;
  return DTSGB_OK;
}

DTSGB_API int dtsgb_pipeline_run_grad(dtsgb_pipeline_t p, int color_space,
                                      const void* const* rgba, const float* const* target,
                                      const float* const* conf,
                                      const dtsgb_filter_params* filter,
                                      const dtsgb_optimize_params* optimize,
                                      const float* const* grad_out, float* const* out_v,
                                      float* const* grad_target,
                                      float* const* grad_confidence) {
  if (!p || !rgba || !target || !filter || !optimize || !grad_out || !out_v)
    return fail(DTSGB_ERR_INVALID_ARGUMENT, "null argument");
  int st = DTSGB_OK;
  size_t k = 0;
  for (; k < p->chunk.size() && !st; ++k) {
    dtsgb_batch_t b = p->chunk[k];
    const int f = p->first[k];
    if (!b->grad) st = dtsgb_batch_enable_grad(b, 1, 0);
    if (!st)
      st = batch_upload(b, color_space, rgba + f, target + f, conf ? conf + f : nullptr,
                        cudaMemcpyHostToDevice, false);
    if (!st) st = dtsgb_batch_solve_dts(b, filter, optimize, -1.f);
    if (!st) st = batch_download(b, 0, out_v + f, cudaMemcpyDeviceToHost, false);
    if (!st)
      st = batch_backward(b, grad_out + f, grad_target ? grad_target + f : nullptr,
                          grad_confidence ? grad_confidence + f : nullptr,
                          cudaMemcpyHostToDevice, cudaMemcpyDeviceToHost, false);
  }
  for (size_t j = 0; j < k; ++j) {
    const cudaError_t e = cudaStreamSynchronize(p->chunk[j]->stream);
    if (e != cudaSuccess && !st) st = cuda_fail(e, "cudaStreamSynchronize");
  }
  return st;
}

DTSGB_API int dtsgb_pipeline_chunks(dtsgb_pipeline_t p) {
  return p ? (int)p->chunk.size() : 0;
}

DTSGB_API int dtsgb_pipeline_batch(dtsgb_pipeline_t p, int k, dtsgb_batch_t* out) {
  if (!p || !out || k < 0 || k >= (int)p->chunk.size())
    return fail(DTSGB_ERR_INVALID_ARGUMENT, "no such chunk");
  *out = p->chunk[k];
  return DTSGB_OK;
}

DTSGB_API int dtsgb_pipeline_run(dtsgb_pipeline_t p, int color_space,
                                 const void* const* rgba, const float* const* target,
                                 const float* const* conf,
                                 const dtsgb_filter_params* filter,
                                 const dtsgb_optimize_params* optimize,
                                 float overwrite_target_above_conf,
                                 const dtsgb_hfbs_params* hfbs, float* const* out_dts,
                                 float* const* out_hfbs) {
  if (!p || !rgba || !target) return fail(DTSGB_ERR_INVALID_ARGUMENT, "null argument");
  const bool dts = filter && optimize;
  if ((dts && !out_dts) || (hfbs && !out_hfbs))
    return fail(DTSGB_ERR_INVALID_ARGUMENT, "null output array");
  int st = DTSGB_OK;
  size_t k = 0;
  for (; k < p->chunk.size() && !st; ++k) {
    dtsgb_batch_t b = p->chunk[k];
    const int f = p->first[k];
    st = batch_upload(b, color_space, rgba + f, target + f, conf ? conf + f : nullptr,
                      cudaMemcpyHostToDevice, false);
    if (!st && dts)
      st = dtsgb_batch_solve_dts(b, filter, optimize, overwrite_target_above_conf);
    if (!st && hfbs) st = dtsgb_batch_solve_hfbs(b, hfbs);
    if (!st && dts) st = batch_download(b, 0, out_dts + f, cudaMemcpyDeviceToHost, false);
    if (!st && hfbs) st = batch_download(b, 1, out_hfbs + f, cudaMemcpyDeviceToHost, false);
  }
  // wait for every chunk enqueued so far, also after a failure (the host
  // buffers must not be in use when this returns)
  for (size_t j = 0; j < k; ++j) {
    const cudaError_t e = cudaStreamSynchronize(p->chunk[j]->stream);
    if (e != cudaSuccess && !st) st = cuda_fail(e, "cudaStreamSynchronize");
  }
  return st;
}

}  // extern "C"
