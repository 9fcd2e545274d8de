// Pinned host memory for results (crane_b200_host_alloc / _free): copies into it run at the link's rate and need no second copy by the host.  us of a copy into pinned /
// pageable memory: 64 KB 11 / 18, 1 MB 29 / 83, 8 MB 157 / 472, 32 MB 601 / 1980 and more (a Python call for a row of 8 KB 19 / 24, of 593 KB 30 / 66).
// Pinning itself takes far longer than it saves one call (cudaHostAlloc of 1 MB 2.2 ms, of 16 MB 12 ms, freeing 0.4 to 1.8 ms), so no call pins.  ONE range of up to SIZE
// bytes, in huge pages where the system has them, is registered by the first request while a handle is open -- the Python engine makes it as it opens -- as far as its
// handles' results need (ms: 2 MB 0.8, 8 MB 1.7, 64 MB 9; to give them back 0.4 to 1.9), and further when a handle that needs more has opened.  Results are pieces of it, the
// smallest free stretch that holds them.  What does not fit gets ordinary memory from the caller, as does what comes when programs have kept the whole range.  It goes back with
// the last handle or, where pieces are still out, with the last of those.  Its pages are private ones: a forked process has copies of its own, where pages of cudaHostAlloc are
// shared and would show it what later calls of its parent write.  us of a new handle's first pass / of later ones: 32 sequences' round over 8192 logits 940 / 862
// (ordinary memory 1030 / 965, buffers pinned one by one 3400 to 10 000 / 865), one token over 151 936 four times 3300 / 2595 (3540 / 2748, 5000 to 8000 / 2600), an image's
// features 8300 / 3380 (9200 / 3880, 18 000 / 3350).
#pragma once

#include <cuda_runtime.h>
#include <sys/mman.h>

#include <algorithm>
#include <cstddef>
#include <map>
#include <mutex>
#include <set>
#include <thread>

namespace cb {

class HostPool {
public:
    static constexpr size_t SIZE = (size_t)64 << 20, PIECE = 4096, LEAST = (size_t)2 << 20;
    static HostPool& get() { static HostPool* p = new HostPool; return *p; }       // (never destroyed: arrays may outlive static objects)

    void* take(size_t bytes) {
        if (bytes == 0 || bytes > SIZE) return nullptr;
        const size_t n = (bytes + PIECE - 1) / PIECE * PIECE;
        std::lock_guard<std::mutex> g(mu_);
        if (handles_ == 0) return nullptr;
        if (reserved_ < want_ && !tried_) { tried_ = true; reserve(); }
        auto best = free_.end();
        for (auto it = free_.begin(); it != free_.end(); ++it)
            if (it->second >= n && (best == free_.end() || it->second < best->second)) best = it;
        if (best == free_.end()) return nullptr;
        const size_t at = best->first, left = best->second - n;
        out_[at] = n;
        free_.erase(best);
        if (left) free_[at + n] = left;
        return base_ + at;
    }
    bool give(void* p) {
        std::lock_guard<std::mutex> g(mu_);
        const char* c = static_cast<const char*>(p);
        if (!base_ || c < base_ || c >= base_ + SIZE) return false;
        auto it = out_.find((size_t)(c - base_));
        if (it == out_.end()) return false;
        auto f = free_.emplace(it->first, it->second).first;
        out_.erase(it);
        auto next = std::next(f);
        if (next != free_.end() && f->first + f->second == next->first && !parts_.count(next->first)) { f->second += next->second; free_.erase(next); }
        if (f != free_.begin()) {
            auto prev = std::prev(f);
            if (prev->first + prev->second == f->first && !parts_.count(f->first)) { prev->second += f->second; free_.erase(f); }
        }
        if (handles_ == 0 && out_.empty()) release();
        return true;
    }
    // `want`: bytes of results that the handle's programs hold at a time
    void opened(int device, size_t want) {
        std::lock_guard<std::mutex> g(mu_);
        ++handles_;
        device_ = device; tried_ = false;
        want_ = std::max(want_, std::min(std::max((want + LEAST - 1) / LEAST * LEAST, LEAST), SIZE));
    }
    void closed() { std::lock_guard<std::mutex> g(mu_); if (--handles_ == 0 && out_.empty()) release(); }

private:
    // On a thread of its own, with a handle's device: the caller's has its current device and context left as they are (a new thread's are GPU 0 and none), and a stream
    // that another thread is capturing does not forbid it.
    template <typename F> static void aside(int device, F&& f) {
        std::thread([&] {
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
            if (cudaThreadExchangeStreamCaptureMode(&mode) == cudaSuccess && cudaSetDevice(device) == cudaSuccess) f();
        }).join();
    }
    void reserve() {
        if (!base_) {
            void* p = mmap(nullptr, SIZE, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
            if (p == MAP_FAILED) return;
            madvise(p, SIZE, MADV_HUGEPAGE);
            base_ = static_cast<char*>(p);
            reserved_on_ = device_;
        }
        const size_t n = want_ - reserved_;
        bool ok = false;
        try { aside(reserved_on_, [&] { ok = cudaHostRegister(base_ + reserved_, n, cudaHostRegisterPortable) == cudaSuccess; }); } catch (const std::exception&) {}
        if (!ok) return;
        parts_.insert(reserved_);
        free_[reserved_] = n;
        reserved_ = want_;
    }
    void release() {
        want_ = 0;
        if (!base_) return;
        size_t left = parts_.size();
        try { aside(reserved_on_, [&] { for (size_t at : parts_) left -= cudaHostUnregister(base_ + at) == cudaSuccess; }); } catch (const std::exception&) {}
        if (left == 0) munmap(base_, SIZE);                  // (else it stays as it is, registered, and is not used again)
        base_ = nullptr;
        reserved_ = 0;
        parts_.clear();
        free_.clear();
    }
    std::mutex mu_;
    char* base_ = nullptr;
    std::set<size_t> parts_;                    // where the stretches registered one by one begin: no piece lies in two
    std::map<size_t, size_t> free_, out_;       // offset -> length; free stretches have pieces that are out, or such a border, between them
    size_t want_ = 0, reserved_ = 0;
    int handles_ = 0, device_ = 0, reserved_on_ = 0;
    bool tried_ = false;                        // one attempt per handle opened
};

}  // namespace cb
