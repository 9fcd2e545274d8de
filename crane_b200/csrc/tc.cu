// Host side of the tensor-core kernels.  See tc.cuh.
#include "tc.cuh"

#include <mutex>
#include <unordered_map>

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
    const void* base; uint64_t rows, cols, ld; uint32_t box_rows, box_cols; int swizzle, type;
    bool operator==(const TmapKey& o) const {
        return base == o.base && rows == o.rows && cols == o.cols && ld == o.ld && box_rows == o.box_rows && box_cols == o.box_cols && swizzle == o.swizzle && type == o.type;
    }
};
struct TmapKeyHash {
    size_t operator()(const TmapKey& k) const {
        size_t h = std::hash<const void*>()(k.base);
        for (uint64_t v : {k.rows, k.cols, k.ld, (uint64_t)k.box_rows, (uint64_t)k.box_cols, (uint64_t)(k.swizzle * 64 + k.type)}) h = h * 1000003u ^ std::hash<uint64_t>()(v);
        return h;
    }
};
bool tc_tmap(CUtensorMap* map, const void* base, CUtensorMapDataType type, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows, uint32_t box_cols,
             CUtensorMapSwizzle swizzle) {
    static std::unordered_map<TmapKey, CUtensorMap, TmapKeyHash> cache;
    static std::mutex mu;
    const TmapKey key{base, rows, cols, ld, box_rows, box_cols, (int)swizzle, (int)type};
    {
        std::lock_guard<std::mutex> g(mu);
        auto it = cache.find(key);
        if (it != cache.end()) { *map = it->second; return true; }
    }
    PFN_encodeTiled enc = get_encode_fn();
    if (!enc) return false;
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {ld * (type == CU_TENSOR_MAP_DATA_TYPE_FLOAT32 ? 4 : 2)};
    cuuint32_t box[2] = {box_cols, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, type, 2, const_cast<void*>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return false;
    std::lock_guard<std::mutex> g(mu);
    if (cache.size() > 8192) cache.clear();
    cache.emplace(key, *map);
    return true;
}

int tc_device_sms() {
    static int sms[CB_MAX_DEV] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= CB_MAX_DEV) return 148;
    if (!sms[dev]) { int v = 0; cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev); sms[dev] = v > 0 ? v : 148; }
    return sms[dev];
}

__global__ void expire_wait_kernel(int* err) {
    __shared__ uint64_t bar;
    __shared__ int gave_up;
    gave_up = 0;
    mbar_init(&bar, 1);
    fence_barrier_init();
    const TcWaitT<2000000> wait{&gave_up, err};
    wait(&bar, 0);
    wait(&bar, 0);                  // (given up: returns at once)
}
int tc_expire_wait(cudaStream_t st) {
    int* err = nullptr;
    if (const int e = tc_err_word(st, &err)) return e;
    expire_wait_kernel<<<1, 1, 0, st>>>(err);
    return (int)cudaGetLastError();
}

__global__ void __cluster_dims__(2, 1, 1) expire_wait_pair_kernel(int* err) {
    __shared__ uint64_t bar;
    __shared__ int gave_up;
    const uint32_t rank = cluster_rank();
    gave_up = 0;
    mbar_init(&bar, 1);
    fence_barrier_init();
    cluster_sync_all();
    const uint32_t peer = peer_smem(&gave_up, rank ^ 1);
    if (rank == 1) { const TcWaitT<2000000> wait{&gave_up, err, peer}; wait(&bar, 0); }
    else { const TcWait wait{&gave_up, err, peer}; wait(&bar, 0); }        // (4 s by itself; the partner's word ends it)
    cluster_sync_all();
    const TcWait both{&gave_up, err, peer};
    both(&bar, 0);                  // (given up: returns at once in either)
    both.drain();
}
int tc_expire_wait_pair(cudaStream_t st) {
    int* err = nullptr;
    if (const int e = tc_err_word(st, &err)) return e;
    expire_wait_pair_kernel<<<2, 1, 0, st>>>(err);
    return (int)cudaGetLastError();
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
