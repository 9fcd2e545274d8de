// Host side of the tensor-core kernels.  See tc.cuh.
#include "tc.cuh"
#include "gemm.cuh"

#include <algorithm>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace cb {

typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static PFN_encodeTiled get_encode_fn() {
    static PFN_encodeTiled fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_encodeTiled>(p);
    });
    return fn;
}

struct TmapKey {
    const void* base; uint64_t rows, cols, ld; uint32_t box_rows, box_cols; int swizzle;
    bool operator==(const TmapKey& o) const {
        return base == o.base && rows == o.rows && cols == o.cols && ld == o.ld && box_rows == o.box_rows && box_cols == o.box_cols && swizzle == o.swizzle;
    }
};
struct TmapKeyHash {
    size_t operator()(const TmapKey& k) const {
        size_t h = std::hash<const void*>()(k.base);
        for (uint64_t v : {k.rows, k.cols, k.ld, (uint64_t)k.box_rows, (uint64_t)k.box_cols, (uint64_t)k.swizzle}) h = h * 1000003u ^ std::hash<uint64_t>()(v);
        return h;
    }
};
bool tc_tmap_16(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows, uint32_t box_cols, CUtensorMapSwizzle swizzle) {
    static std::unordered_map<TmapKey, CUtensorMap, TmapKeyHash> cache;
    static std::mutex mu;
    const TmapKey key{base, rows, cols, ld, box_rows, box_cols, (int)swizzle};
    {
        std::lock_guard<std::mutex> g(mu);
        auto it = cache.find(key);
        if (it != cache.end()) { *map = it->second; return true; }
    }
    PFN_encodeTiled enc = get_encode_fn();
    if (!enc) return false;
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {ld * 2};
    cuuint32_t box[2] = {box_cols, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return false;
    std::lock_guard<std::mutex> g(mu);
    if (cache.size() > 8192) cache.clear();
    cache.emplace(key, *map);
    return true;
}

static std::mutex g_scratch_mu;
static std::unordered_map<uint64_t, TcScratch> g_scratch;
static uint64_t scratch_key(cudaStream_t st) { int dev = 0; cudaGetDevice(&dev); return ((uint64_t)(uintptr_t)st << 6) ^ (uint64_t)dev; }

// Error words of streams: blocks of 1024 in pinned memory, handed out and taken back under g_scratch_mu (pinning a page per stream costs a handle's
// first call milliseconds, giving it back a device synchronisation)
static std::vector<int*> g_err_free;
static int* take_err_word() {
    if (g_err_free.empty()) {
        int* block = nullptr;
        if (cudaHostAlloc((void**)&block, 1024 * sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) { cudaGetLastError(); return nullptr; }
        for (int i = 1023; i >= 0; --i) { block[i] = 0; g_err_free.push_back(block + i); }
    }
    int* w = g_err_free.back();
    g_err_free.pop_back();
    return w;
}

int tc_scratch_get(cudaStream_t st, size_t ws_floats, int n_counters, TcScratch* out) {
    std::lock_guard<std::mutex> g(g_scratch_mu);
    TcScratch& sc = g_scratch[scratch_key(st)];
    if (!sc.err) {
        sc.err = take_err_word();
        if (!sc.err) return (int)cudaErrorMemoryAllocation;
    }
    if (sc.ws_floats < ws_floats || sc.n_counters < n_counters) {
        // (growing: the old buffers may still be in use by kernels in flight on this stream)
        if (sc.ws || sc.counters) { cudaStreamSynchronize(st); cudaFree(sc.ws); cudaFree(sc.counters); }
        sc.ws = nullptr; sc.counters = nullptr;
        const size_t want = std::max(ws_floats, sc.ws_floats);
        const int wantc = std::max(n_counters, std::max(sc.n_counters, 4096));
        sc.ws_floats = 0; sc.n_counters = 0;
        if (cudaMalloc(&sc.ws, want * sizeof(float)) != cudaSuccess) { sc.ws = nullptr; return (int)cudaErrorMemoryAllocation; }
        if (cudaMalloc(&sc.counters, (size_t)wantc * sizeof(int)) != cudaSuccess) { cudaFree(sc.ws); sc.ws = nullptr; sc.counters = nullptr; return (int)cudaErrorMemoryAllocation; }
        sc.ws_floats = want; sc.n_counters = wantc;
        if (cudaMemsetAsync(sc.counters, 0, (size_t)sc.n_counters * sizeof(int), st) != cudaSuccess) return (int)cudaGetLastError();
    }
    *out = sc;
    return 0;
}
bool tc_take_wait_error(cudaStream_t st) {
    std::lock_guard<std::mutex> g(g_scratch_mu);
    auto it = g_scratch.find(scratch_key(st));
    if (it == g_scratch.end() || !it->second.err || !*reinterpret_cast<volatile int*>(it->second.err)) return false;
    *it->second.err = 0;
    return true;
}
void gemm_release_stream(cudaStream_t st) {
    std::lock_guard<std::mutex> g(g_scratch_mu);
    auto it = g_scratch.find(scratch_key(st));
    if (it == g_scratch.end()) return;
    cudaFree(it->second.ws); cudaFree(it->second.counters);
    if (it->second.err) { *it->second.err = 0; g_err_free.push_back(it->second.err); }
    g_scratch.erase(it);
}
int tc_device_sms() {
    static int sms[CB_MAX_DEV] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= CB_MAX_DEV) return 148;
    if (!sms[dev]) { int v = 0; cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev); sms[dev] = v > 0 ? v : 148; }
    return sms[dev];
}

__global__ void __launch_bounds__(256, 1) cluster_probe_kernel() {}
int tc_max_clusters(int cl) {
    static std::mutex mu;
    static int known[CB_MAX_DEV][9] = {};
    int dev = 0;
    if (cl < 2 || cl > 8 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= CB_MAX_DEV) return 0;
    std::lock_guard<std::mutex> g(mu);
    if (!known[dev][cl]) {
        constexpr int SMEM = 208 * 1024;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(cl); cfg.blockDim = dim3(256); cfg.dynamicSmemBytes = SMEM;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = cl; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr; cfg.numAttrs = 1;
        int n = 0;
        if (cudaFuncSetAttribute(cluster_probe_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, cluster_probe_kernel, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
        known[dev][cl] = n + 1;
    }
    return known[dev][cl] - 1;
}

}  // namespace cb
