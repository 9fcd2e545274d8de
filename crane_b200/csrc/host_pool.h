// Pinned host memory for results (crane_b200_host_alloc / _free): copies into it run at the link's rate and need no second copy by the host.
// A copy of 1 MB into pageable memory took 20 us on the link and another 80 to 100 in the driver's staging.  us a call, pageable / pinned: two decode rounds of 32
// sequences over 8192 logits 949 / 848 (dense, two layers), 625 / 532 (Q4_K_M, one); four tokens over 151 936 logits 2740 / 2597; the features
// of an image, 6.4 MB, 3668 / 3367.  Pinning costs 50 us and more, so returned buffers are kept, in powers of two; what is out and what is kept together stay under
// CAP, whatever programs hold on to, and the kept ones go back when the last handle is destroyed.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace cb {

class HostPool {
public:
    static constexpr int MIN_LOG = 12, MAX_LOG = 25;                    // 4 KB .. 32 MB
    static constexpr size_t CAP = (size_t)64 << 20;
    static HostPool& get() { static HostPool* p = new HostPool; return *p; }       // (never destroyed: arrays may outlive static objects)

    void* take(size_t bytes) {
        int c = MIN_LOG;
        while (((size_t)1 << c) < bytes) if (++c > MAX_LOG) return nullptr;
        std::lock_guard<std::mutex> g(mu_);
        if (handles_ == 0) return nullptr;
        void* p = nullptr;
        if (!free_[c - MIN_LOG].empty()) { p = free_[c - MIN_LOG].back(); free_[c - MIN_LOG].pop_back(); }
        else {
            if (held_ + ((size_t)1 << c) > CAP) trim();
            if (held_ + ((size_t)1 << c) > CAP) return nullptr;
            if (cudaHostAlloc(&p, (size_t)1 << c, cudaHostAllocPortable) != cudaSuccess) { cudaGetLastError(); return nullptr; }
            held_ += (size_t)1 << c;
        }
        out_[p] = c;
        return p;
    }
    bool give(void* p) {
        std::lock_guard<std::mutex> g(mu_);
        auto it = out_.find(p);
        if (it == out_.end()) return false;
        const int c = it->second;
        out_.erase(it);
        if (handles_ > 0) free_[c - MIN_LOG].push_back(p);
        else drop(p, c);
        return true;
    }
    void opened() { std::lock_guard<std::mutex> g(mu_); ++handles_; }
    void closed() { std::lock_guard<std::mutex> g(mu_); if (--handles_ == 0) trim(); }
    size_t held() { std::lock_guard<std::mutex> g(mu_); return held_; }

private:
    void drop(void* p, int c) { cudaFreeHost(p); held_ -= (size_t)1 << c; }
    void trim() {
        for (int i = 0; i <= MAX_LOG - MIN_LOG; ++i) {
            for (void* p : free_[i]) drop(p, i + MIN_LOG);
            free_[i].clear();
        }
    }
    std::mutex mu_;
    std::vector<void*> free_[MAX_LOG - MIN_LOG + 1];
    std::unordered_map<void*, int> out_;
    size_t held_ = 0;       // bytes out and kept
    int handles_ = 0;
};

}  // namespace cb
