// Host side of the TMA staging (tma.cuh): tensor-map encoding through the
// driver entry point resolved at run time (no link against libcuda), and
// the per-owner cache of device tables of tensor maps.
#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>
#include <string>

#include "../../include/dtsgb.h"
#include "tma.cuh"

namespace dtsgb {
namespace {

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, []() {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000,
                                         cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    else
      (void)cudaGetLastError();
  });
  return fn;
}

}  // namespace

int tma_encode_grid(CUtensorMap* out, const void* base, const TmaGrid& g, int bx, int by,
                    int bl) {
  auto fn = encode_fn();
  if (!fn) return fail(DTSGB_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled unavailable");
  if (bx <= 0 || bx > 256 || by <= 0 || by > 256 || bl <= 0 || bl > 256 ||
      (bx * 4) % 16 != 0 || ((uintptr_t)base & 15) != 0 || (g.px * 4) % 16 != 0)
    return fail(DTSGB_ERR_UNSUPPORTED, "grid or box outside the TMA limits");
  const cuuint64_t dims[3] = {(cuuint64_t)g.gx, (cuuint64_t)g.gy, (cuuint64_t)g.gl};
  const cuuint64_t strides[2] = {(cuuint64_t)g.px * 4, (cuuint64_t)g.px * g.gy * 4};
  const cuuint32_t box[3] = {(cuuint32_t)bx, (cuuint32_t)by, (cuuint32_t)bl};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims,
                        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return fail(DTSGB_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
  return DTSGB_OK;
}

// No synchronous copies inside a capture: the caller then stages by loads.
static bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cs) != cudaSuccess) {
    (void)cudaGetLastError();
    return true;
  }
  return cs != cudaStreamCaptureStatusNone;
}

TmaCache::~TmaCache() { clear(); }

// One device allocation and one copy for the tables of all keys.
bool TmaCache::upload(const std::vector<CUtensorMap>& maps, const std::vector<Key>& keys) {
  CUtensorMap* d = nullptr;
  if (cudaMalloc((void**)&d, sizeof(CUtensorMap) * maps.size()) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  if (upload_table(d, maps.data(), sizeof(CUtensorMap) * maps.size()) != cudaSuccess) {
    (void)cudaGetLastError();
    cudaFree(d);
    return false;
  }
  allocs_.push_back(d);
  const size_t n = maps.size() / keys.size();
  for (size_t k = 0; k < keys.size(); ++k) tables_[keys[k]] = d + k * n;
  return true;
}

const CUtensorMap* TmaCache::find(const Key& key) const {
  auto it = tables_.find(key);
  return it == tables_.end() ? nullptr : it->second;
}

void TmaCache::prepare_grids(const TmaGrid* grids, int n, const std::vector<const float*>& planes,
                             int bx, int by, int bl, cudaStream_t s) {
  if (!grids || n <= 0) return;
  std::vector<Key> keys;
  std::vector<CUtensorMap> maps;
  for (const float* p : planes) {
    const Key key = std::make_tuple(p, bx, by, 1000 + bl);
    if (!p || find(key) || std::find(keys.begin(), keys.end(), key) != keys.end()) continue;
    keys.push_back(key);
    for (int i = 0; i < n; ++i) {
      maps.emplace_back();
      if (tma_encode_grid(&maps.back(), p + grids[i].off, grids[i], bx, by, bl)) return;
    }
  }
  if (!keys.empty() && !capturing(s)) (void)upload(maps, keys);
}

const CUtensorMap* TmaCache::get_grid(const TmaGrid* grids, int n, const float* plane, int bx,
                                      int by, int bl, cudaStream_t s) {
  if (!grids || n <= 0 || !plane) return nullptr;
  const Key key = std::make_tuple(plane, bx, by, 1000 + bl);
  if (!find(key)) prepare_grids(grids, n, {plane}, bx, by, bl, s);
  return find(key);
}

void TmaCache::clear() {
  for (CUtensorMap* d : allocs_) cudaFree(d);
  allocs_.clear();
  tables_.clear();
}

}  // namespace dtsgb
