// Tensor-map encoding for the TMA pencil kernels.
//
// cuTensorMapEncodeTiled is a driver entry point; it is fetched through the
// runtime (cudaGetDriverEntryPoint) so the library does not link libcuda and
// still loads on hosts without a GPU driver.  Encoded maps are cached by every
// parameter they encode (base address, extents, element size, box), so a cached
// map is valid for any buffer that matches its key, including a freed and
// re-allocated one at the same address.
#include <cudaTypedefs.h>

#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>

#include "kernels.h"

namespace sb200 {

namespace {

using Key = std::tuple<uintptr_t, int64_t, int64_t, int64_t, int, int, int>;

std::mutex g_mu;
std::map<Key, std::unique_ptr<CUtensorMap>>* g_cache = nullptr;
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;

PFN_cuTensorMapEncodeTiled_v12000 encoder() {
    if (!g_encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }
    return g_encode;
}

}  // namespace

namespace {

// Encodes (or takes from the cache) a map of `rank` dimensions: extents n, line strides
// in bytes of dimensions 1.., the box.
int cached_map(CUtensorMap* out, const Key& key, const void* base, int rank, const int64_t* n,
               const int64_t* stride, int esize, const cuuint32_t* box) {
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_cache) g_cache = new std::map<Key, std::unique_ptr<CUtensorMap>>();
    auto it = g_cache->find(key);
    if (it != g_cache->end()) {
        *out = *it->second;
        return 0;
    }

    auto enc = encoder();
    if (!enc) return -1;
    if (g_cache->size() > 4096) g_cache->clear();  // bound host memory for long sessions

    auto map = std::make_unique<CUtensorMap>();
    std::memset(map.get(), 0, sizeof(CUtensorMap));
    cuuint64_t dims[3], strides[2];
    for (int d = 0; d < rank; ++d) dims[d] = static_cast<cuuint64_t>(n[d]);
    for (int d = 0; d + 1 < rank; ++d) strides[d] = static_cast<cuuint64_t>(stride[d]);
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUtensorMapDataType dt =
        esize == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT16;
    const CUresult r = enc(map.get(), dt, rank, const_cast<void*>(base), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return static_cast<int>(r);
    *out = *map;
    (*g_cache)[key] = std::move(map);
    return 0;
}

}  // namespace

int tensor_map_3d(CUtensorMap* out, const void* base, int64_t nx, int64_t ny, int64_t nz,
                  int esize, int box_x, int box_y) {
    const int64_t n[3] = {nx, ny, nz}, stride[2] = {nx * esize, nx * ny * esize};
    const cuuint32_t box[3] = {static_cast<cuuint32_t>(box_x), static_cast<cuuint32_t>(box_y), 1};
    return cached_map(out, Key{reinterpret_cast<uintptr_t>(base), nx, ny, nz, esize, box_x, box_y},
                      base, 3, n, stride, esize, box);
}

int tensor_map_rows4(CUtensorMap* out, const void* base, int64_t nx, int64_t rows, int box_x,
                     int box_y) {
    const int64_t n[2] = {4 * nx, rows / 4}, stride[1] = {16 * nx};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(box_x), static_cast<cuuint32_t>(box_y)};
    return cached_map(out, Key{reinterpret_cast<uintptr_t>(base), nx, rows, 0, 4, box_x, box_y}, base,
                      2, n, stride, 4, box);
}

}  // namespace sb200
