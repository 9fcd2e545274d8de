// Host test of the per-stream scratch (crane_b200/csrc/tc_scratch.cu) against a fake of the CUDA calls it makes: addresses that a captured graph may
// hold stay allocated while the stream lives, whatever is asked for later, and everything is given back with the stream.
#include "../../crane_b200/csrc/tc_scratch.cu"

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>

static std::map<void*, size_t> live;
static size_t fail_above = (size_t)-1;
static int fills_on_user_streams = 0;
static int fake_stream;                                     // the fake of every stream that the scratch makes for itself
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
    if (n > fail_above) return cudaErrorMemoryAllocation;
    *p = malloc(n); live[*p] = n; return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (p && !live.erase(p)) { printf("freed twice or never allocated\n"); exit(1); }
    free(p); return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)&fake_stream; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { if (s != (cudaStream_t)&fake_stream) ++fills_on_user_streams; return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
    if (s != (cudaStream_t)&fake_stream) ++fills_on_user_streams;
    memset(p, v, n); return cudaSuccess;
}
}

#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
    using namespace cb;
    cudaStream_t a = (cudaStream_t)0x1000, b = (cudaStream_t)0x2000;
    int* err = nullptr;
    CHECK(tc_err_word(a, &err) == 0 && err && live.empty());                  // no workspace for a kernel that shares nothing
    TcScratch first, s;
    CHECK(tc_scratch_get(a, 128, &first) == 0 && first.err == err);
    for (int i = 0; i < 4096; ++i) CHECK(first.counters[i] == 0);
    int* at = first.counters;
    size_t largest = 0;
    for (int n : {4096, 4097, 100, 9000, 33000, 5}) {                         // a longer prompt, a short one, ...
        CHECK(tc_scratch_get(a, n, &s) == 0);
        CHECK(s.ws == first.ws && live.count(first.ws));
        CHECK(live.count(first.counters) && live.count(at));                 // what an earlier capture holds is still there
        CHECK(live[s.counters] >= (size_t)n * sizeof(int));
        for (size_t i = 0; i < live[s.counters] / sizeof(int); ++i) CHECK(s.counters[i] == 0);
        at = s.counters;
        largest = live[at];
    }
    size_t counters = 0;
    for (auto& p : live) if (p.first != (void*)first.ws) counters += p.second;
    CHECK(counters < 2 * largest);
    CHECK(fills_on_user_streams == 0);                                       // (they would be captured)
    CHECK(tc_scratch_get(b, 10, &s) == 0 && s.ws != first.ws && s.counters != first.counters && s.err != err);
    *err = 1;
    CHECK(!tc_take_wait_error(b) && tc_take_wait_error(a) && !tc_take_wait_error(a));
    fail_above = 1 << 20;                                                    // out of memory: what there is stays usable
    CHECK(tc_scratch_get(a, 1 << 22, &s) != 0);
    CHECK(tc_scratch_get(a, 33000, &s) == 0 && s.counters == at);
    tc_scratch_release(a);
    tc_scratch_release(b);
    tc_scratch_release(b);
    CHECK(live.empty());
    printf("tc_scratch: ok\n");
    return 0;
}
