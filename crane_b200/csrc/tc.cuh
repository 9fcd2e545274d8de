// tcgen05 / TMA / mbarrier wrappers shared by the tensor-core kernels, and the host side they share: encoded tensor maps and the per-stream
// scratch (tc_scratch.h).
#pragma once

#include <cuda.h>
#include "common.cuh"
#include "tc_scratch.h"

namespace cb {

// ---- bounded waits ---------------------------------------------------------------------
// A wait that runs out (4 s at 1.9 GHz: a wait in these kernels is for a copy or an MMA of its own CTA, or of either CTA of a pair, or for the end of the kernel ahead)
// raises the CTA's `gave_up` word in shared memory, with it that of the other CTA of a pair, and the stream's error word in pinned host memory; every later wait of the
// CTA, or of both, returns at once, the kernel runs to its end with its results discarded, and every call that hands results to the caller reads the word first
// (sync_results in engine.cu) and reports the error.  Results that are left on the device are covered by the call that reads them.
constexpr long long TC_WAIT_CYCLES = 8000000000LL;
constexpr uint32_t TC_NO_PEER = 0xffffffffu;
template <long long LIMIT>
struct TcWaitT {
    volatile int* gave_up;      // shared memory, zeroed before the first wait
    int* err;                   // pinned host memory (tc_err_word), written only when a wait runs out
    uint32_t peer = TC_NO_PEER; // the word of the pair's other CTA (a cluster address), which leaves behind a barrier of both only
    __device__ __forceinline__ void operator()(uint64_t* bar, uint32_t parity) const {
        const uint32_t addr = smem_u32(bar);
        long long t0 = 0;
        for (uint32_t n = 0;; ++n) {
            uint32_t ok;
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(ok) : "r"(addr), "r"(parity) : "memory");
            if (ok) return;
            if ((n & 255u) == 255u) {
                if (*gave_up) return;
                if (!t0) t0 = clock64();
                else if (clock64() - t0 > LIMIT) {
                    *gave_up = 1;
                    if (peer != TC_NO_PEER) asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], 1;" ::"r"(peer) : "memory");
                    *reinterpret_cast<volatile int*>(err) = 1;
                    return;
                }
            }
        }
    }
    // the issuing thread's last act when a wait ran out (in a pair: every thread's of both, behind their last barrier): copies still in flight must not land in a
    // successor's shared memory
    __device__ __forceinline__ void drain() const {
        if (!*gave_up) return;
        const long long t0 = clock64();
        while (clock64() - t0 < 20000000LL) {}
    }
};
using TcWait = TcWaitT<TC_WAIT_CYCLES>;
__device__ __forceinline__ int ld_acquire(const int* p) { int v; asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory"); return v; }
// One lane of a converged warp.  An issuing warp runs its loop as a whole and only its tcgen05 / TMA instructions under this: addresses and descriptors
// stay in uniform registers (measured, 128 x 16 MMAs: 40 cycles each, 52 when a single lane runs the loop).
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
// generic-proxy writes to shared memory (st.shared) become visible to tcgen05.mma / TMA
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ---- PTX wrappers (sm_100a) --------------------------------------------------------------
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1) : "memory");
}
// shared -> global, rows and columns outside the tensor are dropped; and the same with the old values added (f32, in the L2).  One thread issues and commits.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, const void* smem_src, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tma_add_2d(const CUtensorMap* map, const void* smem_src, int c0, int c1) {
    asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];"
                 ::"l"(map), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>      // the sources of all but the last N stores may be rewritten
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {     // A from TMEM
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrives on `bar` when every tcgen05.mma issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// 16 / 8 columns, without the wait: several loads in flight, then one tmem_ld_wait() before their registers are read
__device__ __forceinline__ void tmem_ld16_async(uint32_t taddr, uint32_t* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld8_async(uint32_t taddr, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
        ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
        ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
          "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
          "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---- pairs of CTAs (clusters of two, cta_group::2): one MMA over both SMs, issued by the even CTA -----------------------------------
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
// `p` of this CTA's shared memory in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t peer_smem(const void* p, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_peer(uint32_t bar) { asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory"); }
// into this CTA's shared memory, counted on a barrier of the pair's (a cluster address)
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives on `bar` of both CTAs (the same place in either's shared memory) when every MMA issued so far has completed
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}

// K-major, SWIZZLE_128B shared-memory matrix descriptor (cute::UMMA::SmemDescriptor layout):
// start address >> 4 in [0,14), LBO(=1, ignored for swizzled K-major) in [16,30),
// SBO = 1024 B (8 rows x 128 B) >> 4 in [32,46), version = 1 in [46,48), layout SWIZZLE_128B = 2 in [61,64).
__device__ __forceinline__ uint64_t make_smem_desc_sw128(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// Instruction descriptor (cute::UMMA::InstrDescriptor): D=f32, A=B=bf16, both K-major, M x N.
__host__ __device__ constexpr uint32_t make_idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
// The same for 32-byte rows (16 f16 / bf16): SWIZZLE_32B = 6, SBO = 8 rows x 32 B; the 16-byte half c of row r sits at half c ^ ((r >> 2) & 1).
__device__ __forceinline__ uint64_t make_smem_desc_sw32(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(256 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)6 << 61;
    return d;
}
// A, B = f16 instead of bf16
__host__ __device__ constexpr uint32_t make_idesc_f16(int M, int N) { return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24); }
// 128-byte rows: byte offset of the 16-byte piece c of row r
__device__ __forceinline__ uint32_t sw128_off(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }
// 64- and 32-byte rows
__device__ __forceinline__ uint32_t sw32_off(int r, int c) { return (uint32_t)(r * 32 + ((c ^ ((r >> 2) & 1)) << 4)); }
__device__ __forceinline__ uint32_t sw64_off(int r, int c) { return (uint32_t)(r * 64 + ((c ^ ((r >> 1) & 3)) << 4)); }

// ---- host side (tc.cu) ---------------------------------------------------------------------
// 2-D row-major [rows, cols] of 16- or 32-bit elements with `ld` elements between rows; box = [box_rows, box_cols].  Encoded maps are cached by
// their defining tuple: encoding costs a few microseconds of host time, as much as a small kernel runs.
bool tc_tmap(CUtensorMap* map, const void* base, CUtensorMapDataType type, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows, uint32_t box_cols,
             CUtensorMapSwizzle swizzle);
inline bool tc_tmap_16(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows, uint32_t box_cols, CUtensorMapSwizzle swizzle) {
    return tc_tmap(map, base, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rows, cols, ld, box_rows, box_cols, swizzle);
}
// ... of bf16 in boxes of 64 columns, SWIZZLE_128B
inline bool tc_tmap_bf16(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows) {
    return tc_tmap_16(map, base, rows, cols, ld, box_rows, 64, CU_TENSOR_MAP_SWIZZLE_128B);
}
// launches a kernel whose wait runs out after about a millisecond (for tests of what follows)
int tc_expire_wait(cudaStream_t st);
int tc_expire_wait_pair(cudaStream_t st);      // ... one CTA's of a pair, while the other waits for what never comes
int tc_device_sms();
// clusters of `cl` (2 .. 8) CTAs that the device runs at the same time when a CTA takes a whole SM
int tc_max_clusters(int cl);

// ---- work dealt out along K ------------------------------------------------------------------
// G CTAs share tiles x KB iterations; CTA c owns the iterations [unit * (c * base + min(c, rem)), ...): base or base + 1 units of `unit`
// iterations -- unit = KB deals out whole tiles (nothing is split; where a CTA's j-th lies: sched_place), unit = 1 is stream-K
struct TcSched {
    int tiles_m, tiles_n, KB;      // output tiles and iterations per tile; tile t: sched_place (a linear of few rows, gemm_rows.cu: one row of tiles)
    int G, unit, base, rem;
    int band;                      // rows of tiles that sched_place walks together (tiles_m: all of them)
    float* ws;                     // [2 * G] partial tiles
    int* counters;                 // [tiles] arrivals per tile, zero between launches (the finisher resets its tile)
};
__host__ __device__ inline int sched_start(const TcSched& s, int c) { return s.unit * (c * s.base + (c < s.rem ? c : s.rem)); }
__host__ __device__ inline int sched_owner(const TcSched& s, int it) {       // CTA whose range holds iteration `it`
    const int u = it / s.unit, big = s.rem * (s.base + 1);
    return u < big ? u / (s.base + 1) : s.rem + (u - big) / s.base;
}
// Where tile t of CTA c's range lies.  Whole tiles: the CTA's j-th is number c + j * G, so that the G tiles of a turn are neighbours (a CTA has base tiles, the first rem one
// more: every number below G * base + rem once); numbers run along the rows of a band, then along n, then to the next band.
__host__ __device__ inline void sched_place(const TcSched& s, int c, int t, int& mt, int& nt) {
    if (s.unit == s.KB) t = c + (t - (c * s.base + (c < s.rem ? c : s.rem))) * s.G;
    const int per = s.band * s.tiles_n, b = t / per, r = t - b * per, left = s.tiles_m - b * s.band, w = left < s.band ? left : s.band;
    nt = r / w;
    mt = b * s.band + r - nt * w;
}

}  // namespace cb
