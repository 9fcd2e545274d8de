// See tc_scratch.h.
#include "tc_scratch.h"

#include <cstdint>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace cb {

namespace {
struct StreamScratch {
    float* ws = nullptr;
    std::vector<int*> counters;       // blocks, each larger than the one before; only the last is handed out from now on
    int n_counters = 0;
    int* err = nullptr;
};
std::mutex g_mu;
std::unordered_map<uint64_t, StreamScratch> g_scratch;
uint64_t key_of(cudaStream_t st) { int dev = 0; cudaGetDevice(&dev); return ((uint64_t)(uintptr_t)st << 6) ^ (uint64_t)dev; }

// Error words of streams: blocks of 1024 in pinned memory, handed out and taken back under g_mu (pinning a page per stream costs a handle's
// first call milliseconds, giving it back a device synchronisation)
std::vector<int*> g_err_free;
int* take_err_word() {
    if (g_err_free.empty()) {
        int* block = nullptr;
        if (cudaHostAlloc((void**)&block, 1024 * sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) { cudaGetLastError(); return nullptr; }
        for (int i = 1023; i >= 0; --i) { block[i] = 0; g_err_free.push_back(block + i); }
    }
    int* w = g_err_free.back();
    g_err_free.pop_back();
    return w;
}

// Zeroed by a stream of its own and waited for: on `st`, a fill would become part of a graph that is being captured there
int zeroed_ints(int n, int** out) {
    int* p = nullptr;
    cudaStream_t s = nullptr;
    cudaError_t e = cudaMalloc((void**)&p, (size_t)n * sizeof(int));
    if (e != cudaSuccess) { cudaGetLastError(); return (int)e; }
    e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMemsetAsync(p, 0, (size_t)n * sizeof(int), s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (s) cudaStreamDestroy(s);
    if (e != cudaSuccess) { cudaFree(p); return (int)e; }
    *out = p;
    return 0;
}

int with_err(cudaStream_t st, StreamScratch** out) {       // (under g_mu)
    StreamScratch& sc = g_scratch[key_of(st)];
    if (!sc.err) sc.err = take_err_word();
    *out = &sc;
    return sc.err ? 0 : (int)cudaErrorMemoryAllocation;
}
}  // namespace

int tc_scratch_get(cudaStream_t st, int n_counters, TcScratch* out) {
    std::lock_guard<std::mutex> g(g_mu);
    StreamScratch* sc = nullptr;
    if (const int e = with_err(st, &sc)) return e;
    if (!sc->ws) {
        const cudaError_t e = cudaMalloc((void**)&sc->ws, TC_WS_FLOATS * sizeof(float));
        if (e != cudaSuccess) { cudaGetLastError(); sc->ws = nullptr; return (int)e; }
    }
    if (sc->counters.empty() || sc->n_counters < n_counters) {
        int want = 4096, *p = nullptr;
        while (want < n_counters) want *= 2;
        if (const int e = zeroed_ints(want, &p)) return e;
        sc->counters.push_back(p);
        sc->n_counters = want;
    }
    *out = TcScratch{sc->ws, sc->counters.back(), sc->err};
    return 0;
}

int tc_err_word(cudaStream_t st, int** out) {
    std::lock_guard<std::mutex> g(g_mu);
    StreamScratch* sc = nullptr;
    if (const int e = with_err(st, &sc)) return e;
    *out = sc->err;
    return 0;
}

bool tc_take_wait_error(cudaStream_t st) {
    std::lock_guard<std::mutex> g(g_mu);
    auto it = g_scratch.find(key_of(st));
    if (it == g_scratch.end() || !it->second.err || !*reinterpret_cast<volatile int*>(it->second.err)) return false;
    *it->second.err = 0;
    return true;
}

void tc_scratch_release(cudaStream_t st) {
    std::lock_guard<std::mutex> g(g_mu);
    auto it = g_scratch.find(key_of(st));
    if (it == g_scratch.end()) return;
    cudaFree(it->second.ws);
    for (int* p : it->second.counters) cudaFree(p);
    if (it->second.err) { *it->second.err = 0; g_err_free.push_back(it->second.err); }
    g_scratch.erase(it);
}

}  // namespace cb
