// tcgen05 + TMA GEMM for the prefill / ViT path.  See gemm.cuh for the design notes.
#include "gemm.cuh"
#include "tc.cuh"

#include <algorithm>
#include <cmath>
#include <cstdlib>

namespace cb {

// CRANE_B200_GEMM_BN=64|128|256 pins the tile width, 512 the tiles of CTA pairs (sweeps).  (Clusters of 2 x 2 that share their loads
// did not pay on B200: the L2 already merges concurrent requests for a line from a few CTAs.)
static const int g_gemm_bn = [] { const char* e = getenv("CRANE_B200_GEMM_BN"); return e ? atoi(e) : 0; }();

// =====================================================================================
// Row-per-lane stores of 32 finished columns (bias already added), for the SIMT debugging kernel.
// =====================================================================================
template <int MODE>
__device__ __forceinline__ void epi_store32(const GemmEpi& ep, int m, int n, float* v, bool ok) {
    if (!ok) return;
    if constexpr (MODE == EPI_STORE_F32 || MODE == EPI_RESID_F32) {
        float4* o = reinterpret_cast<float4*>(reinterpret_cast<float*>(ep.out) + (size_t)m * ep.ldo + n);
        float4 x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = MODE == EPI_RESID_F32 ? o[j] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = make_float4(x[j].x + v[4 * j], x[j].y + v[4 * j + 1], x[j].z + v[4 * j + 2], x[j].w + v[4 * j + 3]);
    } else if constexpr (MODE == EPI_SILU_MUL_BF16) {
        const size_t off = (size_t)m * ep.ldo + (n >> 1);
        uint32_t p[8], q[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) split_bf16x2(glu_pair_f(v[4 * j], v[4 * j + 1], ep.glu_limit), glu_pair_f(v[4 * j + 2], v[4 * j + 3], ep.glu_limit), p[j], q[j]);
        bf16* o = reinterpret_cast<bf16*>(ep.out) + off;
        *reinterpret_cast<uint4*>(o) = make_uint4(p[0], p[1], p[2], p[3]);
        *reinterpret_cast<uint4*>(o + 8) = make_uint4(p[4], p[5], p[6], p[7]);
        if (ep.out_lo != nullptr) {
            bf16* ol = reinterpret_cast<bf16*>(ep.out_lo) + off;
            *reinterpret_cast<uint4*>(ol) = make_uint4(q[0], q[1], q[2], q[3]);
            *reinterpret_cast<uint4*>(ol + 8) = make_uint4(q[4], q[5], q[6], q[7]);
        }
    } else {
        const size_t off = (size_t)m * ep.ldo + n;
        bf16* o = reinterpret_cast<bf16*>(ep.out) + off;
        bf16* ol = ep.out_lo != nullptr ? reinterpret_cast<bf16*>(ep.out_lo) + off : nullptr;
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
            uint32_t p[4], q[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                float a = v[j + 2 * t], b = v[j + 2 * t + 1];
                if constexpr (MODE == EPI_GELU_ERF_BF16) { a = gelu_erf_f(a); b = gelu_erf_f(b); }
                else if constexpr (MODE == EPI_GELU_TANH_BF16) { a = gelu_tanh_f(a); b = gelu_tanh_f(b); }
                else if constexpr (MODE == EPI_RELU2_BF16) { a = fmaxf(a, 0.f); b = fmaxf(b, 0.f); a *= a; b *= b; }
                split_bf16x2(a, b, p[t], q[t]);
            }
            *reinterpret_cast<uint4*>(o + j) = make_uint4(p[0], p[1], p[2], p[3]);
            if (ol != nullptr) *reinterpret_cast<uint4*>(ol + j) = make_uint4(q[0], q[1], q[2], q[3]);
        }
    }
}

// =====================================================================================
// Fused epilogue of one warp: 32 rows x 32 accumulator columns at a time (lane = row, as tcgen05.ld delivers them).  The arithmetic (bias, scale, gate,
// activation, bf16 split) runs on the lane's own row; the results go to 2 KB patches of shared memory in TMA's swizzled order without bank
// conflicts, and leave as TMA stores, the residual's as TMA adds: the old values never pass through the SM, rows and columns outside the matrix are dropped by the
// copy engine.  (Row-per-lane stores cost 32 LSU wavefronts per instruction, and reading the residual first put a round trip to the L2 into every
// block of columns.)
// A turn of the loop is 32 columns and is not unrolled further: a CTA with one tile runs this code once or twice, out of a cold instruction cache (64 unrolled
// columns: gate / up of a 77-row turn 26.9 us instead of 25.1), while a turn's own chain (TMEM load, proxy fence, store) is too long for 16
// (784 x 4096 with GELU: 25.5 us, 21.6 with 32).
// A warp has one patch of its own.  The epilogue of a CTA's last segment, which nothing runs beside, has four in the operand ring, free by
// then.  32 KB of own patches instead of 16 measured slower (320 x 6144 x 4096 34.9 us, 32.3 with 16): the kernels before and after a linear want the
// rest of the shared memory.
// =====================================================================================
constexpr int EPI_WARPS = 8;
constexpr int EPI_PATCH = 2048;

__device__ __forceinline__ void epi_linear(const GemmEpi& ep, int m, int M, int n, float* v) {
    if (ep.bias != nullptr) {
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            const float4 b = __ldg(reinterpret_cast<const float4*>(ep.bias + n + j));
            v[j] += b.x; v[j + 1] += b.y; v[j + 2] += b.z; v[j + 3] += b.w;
        }
    }
    if (ep.col_scale != nullptr) {
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            const float4 c = __ldg(reinterpret_cast<const float4*>(ep.col_scale + n + j));
            v[j] *= c.x; v[j + 1] *= c.y; v[j + 2] *= c.z; v[j + 3] *= c.w;
        }
    }
    if (ep.gate != nullptr && m < M) {                  // a lane holds 32 neighbouring columns of its own row
        const float* g = ep.gate + (size_t)m * ep.ldg + n;
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            float4 z = *reinterpret_cast<const float4*>(g + j);
            if (ep.gate_bias != nullptr) { const float4 b = *reinterpret_cast<const float4*>(ep.gate_bias + n + j); z.x += b.x; z.y += b.y; z.z += b.z; z.w += b.w; }
            v[j] *= 1.f / (1.f + expf(-z.x)); v[j + 1] *= 1.f / (1.f + expf(-z.y)); v[j + 2] *= 1.f / (1.f + expf(-z.z)); v[j + 3] *= 1.f / (1.f + expf(-z.w));
        }
    }
}

struct EpiPatch {
    uint8_t* base;
    bool ring;          // four patches, else one
    int n = 0;          // stores so far
    // the next patch, its last store's reads done
    __device__ __forceinline__ uint8_t* take(int lane) const {
        if (lane == 0) { if (ring) tma_store_wait_read<3>(); else tma_store_wait_read<0>(); }
        __syncwarp();
        return base + (ring ? (n & 3) * EPI_PATCH : 0);
    }
    // written by every lane: lane 0 may hand it to the copy engine
    __device__ __forceinline__ void ready() {
        fence_proxy_async();
        __syncwarp();
        ++n;
    }
};
// BN accumulator columns of rows m0 .. m0 + 31, shared by the row quarter's warps (`part` of EPI_WARPS / 4); load(c, v) gives columns 32 c .. 32 c + 31.
// A patch is 16 f32 columns, 32 columns of one bf16 plane, or (gate / up, whose 32 columns are 16 results) 16 of both planes.
template <int MODE, int BN, typename Load>
__device__ __forceinline__ void epi_rows(const GemmEpi& ep, const CUtensorMap& tmO, const CUtensorMap& tmOlo, EpiPatch& patch, int m0, int M, int n0, int N, int part,
                                         int lane, Load&& load) {
    constexpr bool F32 = MODE == EPI_STORE_F32 || MODE == EPI_RESID_F32, GLU = MODE == EPI_SILU_MUL_BF16;
#pragma unroll 1
    for (int c = part; c < BN / 32; c += EPI_WARPS / 4) {
        const int n = n0 + 32 * c;
        if (n >= N) break;
        float v[32];
        load(c, v);
        epi_linear(ep, m0 + lane, M, n, v);
        if constexpr (F32) {
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                uint8_t* p = patch.take(lane);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    *reinterpret_cast<float4*>(p + sw64_off(lane, j)) = make_float4(v[16 * g + 4 * j], v[16 * g + 4 * j + 1], v[16 * g + 4 * j + 2], v[16 * g + 4 * j + 3]);
                patch.ready();
                if (lane == 0) {
                    if constexpr (MODE == EPI_RESID_F32) tma_add_2d(&tmO, p, n + 16 * g, m0);
                    else tma_store_2d(&tmO, p, n + 16 * g, m0);
                    tma_store_commit();
                }
            }
        } else if constexpr (GLU) {
            if (m0 + lane >= M) {                       // rows behind the last are zeros, which the division takes 100 cycles each for
#pragma unroll
                for (int j = 0; j < 32; j += 2) v[j] = 1.f;
            }
            if (ep.glu_limit == 0.f) {                  // (outside the loop: sixteen independent exponentials and divisions)
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = silu_f(v[2 * j]) * v[2 * j + 1];
            } else {
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = glu_pair_f(v[2 * j], v[2 * j + 1], ep.glu_limit);
            }
            uint32_t hi[8], lo[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) split_bf16x2(v[2 * j], v[2 * j + 1], hi[j], lo[j]);
            uint8_t* p = patch.take(lane);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                *reinterpret_cast<uint4*>(p + sw32_off(lane, j)) = make_uint4(hi[4 * j], hi[4 * j + 1], hi[4 * j + 2], hi[4 * j + 3]);
                *reinterpret_cast<uint4*>(p + EPI_PATCH / 2 + sw32_off(lane, j)) = make_uint4(lo[4 * j], lo[4 * j + 1], lo[4 * j + 2], lo[4 * j + 3]);
            }
            patch.ready();
            if (lane == 0) {
                tma_store_2d(&tmO, p, n / 2, m0);
                if (ep.out_lo != nullptr) tma_store_2d(&tmOlo, p + EPI_PATCH / 2, n / 2, m0);
                tma_store_commit();
            }
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                if constexpr (MODE == EPI_GELU_ERF_BF16) v[j] = gelu_erf_f(v[j]);
                else if constexpr (MODE == EPI_GELU_TANH_BF16) v[j] = gelu_tanh_f(v[j]);
                else if constexpr (MODE == EPI_RELU2_BF16) { v[j] = fmaxf(v[j], 0.f); v[j] *= v[j]; }
            }
            uint32_t hi[16], lo[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) split_bf16x2(v[2 * j], v[2 * j + 1], hi[j], lo[j]);
            uint8_t* p = patch.take(lane);
#pragma unroll
            for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(p + sw64_off(lane, j)) = make_uint4(hi[4 * j], hi[4 * j + 1], hi[4 * j + 2], hi[4 * j + 3]);
            patch.ready();
            if (lane == 0) { tma_store_2d(&tmO, p, n, m0); tma_store_commit(); }
            if (ep.out_lo != nullptr) {
                p = patch.take(lane);
#pragma unroll
                for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(p + sw64_off(lane, j)) = make_uint4(lo[4 * j], lo[4 * j + 1], lo[4 * j + 2], lo[4 * j + 3]);
                patch.ready();
                if (lane == 0) { tma_store_2d(&tmOlo, p, n, m0); tma_store_commit(); }
            }
        }
    }
}

// =====================================================================================
// tcgen05 kernel: persistent, stream-K over (tile, k-step) iterations, 384 threads per CTA, one CTA per SM
//   warp 0 : TMA producer (one elected lane)       warp 1 : MMA issuer (one elected lane)
//   warp 2 : TMEM allocator / deallocator           warps 4-11 : epilogue (TMEM lane quadrant = warp % 4, two warps share its columns)
//
// Why stream-K.  At the prefill shapes of this engine (M = 454 text rows, 784 patches) a 128 x BN grid of output tiles is either too
// few CTAs (BN = 256: 32-64 tiles for N = 2048-4096) or, with narrow tiles, bound by operand traffic; so the work can be cut the other way: the iteration space
// tiles x k-steps is dealt out evenly, in order, to min(#SMs, ...) CTAs; a CTA whose range starts or ends inside a tile owns a
// PARTIAL sum of that tile.  Partials go to a workspace; the contributor that arrives last adds them IN CONTRIBUTOR ORDER (so the
// result does not depend on who was last: bitwise reproducible) and runs the fused epilogue.  Nobody ever waits for another CTA.
// The accumulator is double-buffered in TMEM (2 x BN columns): the MMAs of a CTA's next segment run under the epilogue of the last.
// =====================================================================================
constexpr int GEMM_BM = 128;
constexpr int GEMM_BK = 64;
constexpr int GEMM_STAGE_BUDGET = 192 * 1024;
constexpr int GEMM_MAX_CTAS = 160;                 // workspace slots: two partial tiles per CTA

template <int BN, bool SPLIT>
struct GemmCfg {
    static constexpr int A_BYTES = GEMM_BM * GEMM_BK * 2;
    static constexpr int B_BYTES = BN * GEMM_BK * 2;
    static constexpr int STAGE_BYTES = A_BYTES * (SPLIT ? 2 : 1) + B_BYTES;     // [A hi | A lo (SPLIT) | B]
    static constexpr int STAGES = (GEMM_STAGE_BUDGET / STAGE_BYTES) < 8 ? (GEMM_STAGE_BUDGET / STAGE_BYTES) : 8;
    static constexpr int EPI_BYTES = EPI_WARPS * EPI_PATCH;                     // store patches of the epilogue warps
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_BYTES + 1024 /*align*/ + 256 /*barriers*/;
    static constexpr int TMEM_COLS = 2 * BN;
};

// What the epilogue warps do with the accumulators of a CTA's segments.  `cta`: the CTA's place in the schedule, with PER = 2 the pair's, of which this is CTA `rank`;
// every CTA has 128 rows of a tile, partial tiles and counters of its own.
template <int MODE, int BN, int PER, typename Ready, typename Drained>
__device__ __forceinline__ void gemm_epilogue(const GemmEpi& ep, const CUtensorMap& tmO, const CUtensorMap& tmOlo, EpiPatch& patch, uint8_t* ring, int M, int N, const TcSched& sc, int cta,
                                              int rank, int it_begin, int it_end, uint32_t tmem_base, uint64_t* tmem_full_bar, const TcWait& wait, int* last_flag, int q, int part,
                                              int lane, Ready&& first_ready, Drained&& drained) {
    const int KB = sc.KB;
    constexpr int CHUNKS = BN / 32;
    constexpr size_t TILE_F = (size_t)GEMM_BM * BN;
    int seg = 0;
    for (int it = it_begin; it < it_end; ++seg) {
        const int seg_end = min(it_end, (it / KB + 1) * KB);
        const int t = it / KB, kb0 = it % KB, kb1 = kb0 + (seg_end - it);
        int mt, nt;
        sched_place(sc, cta, t, mt, nt);
        const int m0 = (mt * PER + rank) * GEMM_BM + q * 32, n0 = nt * BN;
        const int b = seg & 1;
        const uint32_t acc = tmem_base + (uint32_t)(b * BN) + ((uint32_t)(q * 32) << 16);
        const bool sole = kb0 == 0 && kb1 == KB;
        const int c_first = sched_owner(sc, t * KB), c_last = sched_owner(sc, t * KB + KB - 1);
        // a shared tile whose other contributors have all arrived already is finished without parking this part (read while the MMAs run)
        if (!sole && threadIdx.x == 128) *last_flag = ld_acquire(&sc.counters[t * PER + rank]) == c_last - c_first;
        wait(&tmem_full_bar[b], (seg >> 1) & 1);
        tc_fence_after();
        if (threadIdx.x == 128 && seg == 0) first_ready();
        bool finish = sole;
        if (!sole) {
            named_bar_sync(1, 32 * EPI_WARPS);
            finish = *last_flag;
            if (!finish) {
                // park it.  A 32 x 32 block of (row = lane, column j) is stored as 8 rows of 32 float4: the float4
                // of lane l in row k holds columns 4k .. 4k+3 of row l, so every store / reload instruction moves 512 contiguous bytes
                float* mine = sc.ws + (size_t)((2 * cta + (it == it_begin ? 0 : 1)) * PER + rank) * TILE_F + (size_t)q * CHUNKS * 1024;
#pragma unroll 1
                for (int c = part; c < CHUNKS; c += EPI_WARPS / 4) {
                    uint32_t r[32];
                    tmem_ld32(acc + (uint32_t)(c * 32), r);
                    float4* dst = reinterpret_cast<float4*>(mine + c * 1024) + lane;
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        dst[k * 32] = make_float4(__uint_as_float(r[4 * k]), __uint_as_float(r[4 * k + 1]), __uint_as_float(r[4 * k + 2]), __uint_as_float(r[4 * k + 3]));
                }
                // arrive at the tile; the last of its contributors finishes it
                __threadfence();
                named_bar_sync(1, 32 * EPI_WARPS);
                if (threadIdx.x == 128) *last_flag = atomicAdd(&sc.counters[t * PER + rank], 1) == c_last - c_first;
                named_bar_sync(1, 32 * EPI_WARPS);
                finish = *last_flag;
            }
            if (finish) {
                __threadfence();
                if (threadIdx.x == 128) sc.counters[t * PER + rank] = 0;       // clean for the next launch on this stream
            }
        }
        if (seg_end == it_end) { patch.base = ring; patch.ring = true; }      // every MMA of this CTA has read its operands
        if (finish && m0 < M)
            epi_rows<MODE, BN>(ep, tmO, tmOlo, patch, m0, M, n0, N, part, lane, [&](int c, float* v) {
                tmem_ld32(acc + (uint32_t)(c * 32), reinterpret_cast<uint32_t*>(v));
                if (sole) return;
                // a shared tile: contributor order, whoever came last
                float sum[32];
#pragma unroll
                for (int j = 0; j < 32; ++j) sum[j] = 0.f;
#pragma unroll 1
                for (int cc = c_first; cc <= c_last; ++cc) {
                    if (cc == cta) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) sum[j] += v[j];
                        continue;
                    }
                    const float4* p = reinterpret_cast<const float4*>(sc.ws + (size_t)((2 * cc + (sched_start(sc, cc) < t * KB ? 1 : 0)) * PER + rank) * TILE_F +
                                                                      (size_t)(q * CHUNKS + c) * 1024) + lane;
                    float4 x[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) x[k] = __ldcg(p + k * 32);
#pragma unroll
                    for (int k = 0; k < 8; ++k) { sum[4 * k] += x[k].x; sum[4 * k + 1] += x[k].y; sum[4 * k + 2] += x[k].z; sum[4 * k + 3] += x[k].w; }
                }
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = sum[j];
            });
        tc_fence_before();
        __syncwarp();
        if (lane == 0) drained(b);
        if (!sole) named_bar_sync(1, 32 * EPI_WARPS);             // last_flag is rewritten by the next segment
        it = seg_end;
    }
}

// SPLIT: the activation operand comes as two bf16 planes A = hi + lo (lo = bf16(x - hi), ~16 mantissa bits together); the
// weight tile is fetched once and multiplied by both, accumulating into the same TMEM columns: D = hi.W^T + lo.W^T.
// (Bounds: 384 threads, but no more registers than 512 would leave each: the row kernels beside a linear need some too.)
template <int BN, int MODE, bool SPLIT>
__global__ void __launch_bounds__(512, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmAlo, const __grid_constant__ CUtensorMap tmB,
               const __grid_constant__ CUtensorMap tmO, const __grid_constant__ CUtensorMap tmOlo, GemmEpi ep, int M, int N, int K, TcSched sc, int* err) {
    using Cfg = GemmCfg<BN, SPLIT>;
    constexpr int STAGES = Cfg::STAGES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* epi_smem = smem + STAGES * Cfg::STAGE_BYTES;
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(epi_smem + Cfg::EPI_BYTES);
    uint64_t* empty_bar = full_bar + STAGES;
    uint64_t* tmem_full_bar = empty_bar + STAGES;      // [2] accumulator b complete
    uint64_t* tmem_empty_bar = tmem_full_bar + 2;      // [2] accumulator b drained by the epilogue warps
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty_bar + 2);
    int* last_flag = reinterpret_cast<int*>(tmem_slot + 1);
    int* gave_up = last_flag + 1;
    const TcWait wait{gave_up, err};

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cta = blockIdx.x;
    const int KB = sc.KB;
    const int it_begin = sched_start(sc, cta), it_end = sched_start(sc, cta + 1);
    // optional timeline of this CTA (tools/gemm_probe.py): 8 globaltimer stamps per CTA
    unsigned long long* prof = ep.prof ? ep.prof + 8 * (size_t)cta : nullptr;
    auto stamp = [&](int i) {
        if (prof) { unsigned long long t; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t)); prof[i] = t; }
    };
    if (threadIdx.x == 0) stamp(0);

    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmA);
        if (SPLIT) tma_prefetch_desc(&tmAlo);
        tma_prefetch_desc(&tmB);
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full_bar[b], 1); mbar_init(&tmem_empty_bar[b], EPI_WARPS); }
        *gave_up = 0;
        fence_barrier_init();
    }
    if (warp == 2) { tmem_alloc(tmem_slot, Cfg::TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (threadIdx.x == 0) stamp(1);                 // setup done

    pdl_launch_dependents();                        // the next kernel may begin its own setup / weight prefetch now
    if (warp == 0) {
        if (lane == 0) {
            // A step takes the tensor pipe 130 to 530 ns and the issuing thread should take far less: the tile's coordinates are divided out once per
            // segment, not per step.  (Four integer divisions a step made a step of plain bf16 cost 325 - 420 ns whatever the tile's width; without them 250 with 64 columns, 267
            // with 128, 340 - 420 with 256.)
            constexpr int B_OFF = Cfg::A_BYTES * (SPLIT ? 2 : 1);
            // weights do not depend on the predecessor kernel: their first tiles go out before the dependency wait
            const int npre = ep.w_dynamic ? 0 : min(it_end - it_begin, STAGES);
            int t = it_begin / KB, kb = it_begin - t * KB, mt, nt;
            sched_place(sc, cta, t, mt, nt);
            int n0 = nt * BN;
            for (int i = 0; i < npre; ++i) {
                mbar_arrive_expect_tx(&full_bar[i], Cfg::STAGE_BYTES);
                tma_load_2d(smem + i * Cfg::STAGE_BYTES + B_OFF, &tmB, &full_bar[i], kb * GEMM_BK, n0);
                if (++kb == KB && i + 1 < npre) { kb = 0; sched_place(sc, cta, ++t, mt, nt); n0 = nt * BN; }
            }
            pdl_wait();
            int s = 0, left = npre; uint32_t ph = 0;
            for (int it = it_begin; it < it_end;) {
                t = it / KB;
                sched_place(sc, cta, t, mt, nt);
                const int seg_end = min(it_end, (t + 1) * KB), m0 = mt * GEMM_BM;
                n0 = nt * BN;
                int kc = (it - t * KB) * GEMM_BK;
                for (; it < seg_end; ++it, kc += GEMM_BK) {
                    uint8_t* a_dst = smem + s * Cfg::STAGE_BYTES;
                    if (left > 0) --left;
                    else {
                        wait(&empty_bar[s], ph ^ 1);
                        mbar_arrive_expect_tx(&full_bar[s], Cfg::STAGE_BYTES);
                        tma_load_2d(a_dst + B_OFF, &tmB, &full_bar[s], kc, n0);
                    }
                    tma_load_2d(a_dst, &tmA, &full_bar[s], kc, m0);
                    if (SPLIT) tma_load_2d(a_dst + Cfg::A_BYTES, &tmAlo, &full_bar[s], kc, m0);
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
            }
            wait.drain();
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = make_idesc_bf16(GEMM_BM, BN);
        int s = 0; uint32_t ph = 0;
        int seg = 0;
        for (int it = it_begin; it < it_end; ++seg) {
            const int seg_end = min(it_end, (it / KB + 1) * KB);
            const int b = seg & 1;
            wait(&tmem_empty_bar[b], ((seg >> 1) & 1) ^ 1);           // the epilogue has drained this accumulator (first two: free)
            tc_fence_after();
            const uint32_t acc = tmem_base + (uint32_t)(b * BN);
            for (int i = it; i < seg_end; ++i) {
                wait(&full_bar[s], ph);
                tc_fence_after();
                if (lane == 0 && i == it_begin) stamp(2);             // first operands landed
                const uint32_t a_addr = smem_u32(smem + s * Cfg::STAGE_BYTES);
                const uint64_t adesc = make_smem_desc_sw128(a_addr);
                const uint64_t aldesc = make_smem_desc_sw128(a_addr + Cfg::A_BYTES);
                const uint64_t bdesc = make_smem_desc_sw128(a_addr + Cfg::A_BYTES * (SPLIT ? 2 : 1));
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < GEMM_BK / 16; ++k) {
                        // +32 B per K=16 step inside the 128 B swizzle atom -> +2 in the >>4-encoded start address
                        umma_bf16(acc, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc, (uint32_t)((i != it) | (k != 0)));
                        if (SPLIT) umma_bf16(acc, aldesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc, 1u);
                    }
                    umma_commit(&empty_bar[s]);                       // frees the smem stage once these MMAs retire
                    if (i == seg_end - 1) umma_commit(&tmem_full_bar[b]);         // this segment's accumulator is complete
                }
                __syncwarp();
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
            it = seg_end;
        }
        if (lane == 0) stamp(3);                                      // last MMA issued
    } else if (warp >= 4) {
        if (threadIdx.x == 128) { tma_prefetch_desc(&tmO); tma_prefetch_desc(&tmOlo); }
        pdl_wait();                                 // the epilogue reads / overwrites activations of the predecessor too
        const int q = warp & 3, part = (warp - 4) >> 2;
        EpiPatch patch{epi_smem + (warp - 4) * EPI_PATCH, false};
        gemm_epilogue<MODE, BN, 1>(ep, tmO, tmOlo, patch, smem + (warp - 4) * 4 * EPI_PATCH, M, N, sc, cta, 0, it_begin, it_end, tmem_base, tmem_full_bar, wait, last_flag, q, part, lane,
                                   [&] { stamp(4); }, [&](int b) { mbar_arrive(&tmem_empty_bar[b]); });      // (stamp: first accumulator ready)
        if (lane == 0) tma_store_wait_read<0>();        // (the writes themselves are complete when the grid is)
        if (threadIdx.x == 128) stamp(5);               // this CTA's rows stored
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0) stamp(6);                 // whole CTA done
    if (warp == 2) { tc_fence_after(); tmem_dealloc(tmem_base, Cfg::TMEM_COLS); if (lane == 0) stamp(7); }
}

// =====================================================================================
// The same over pairs of CTAs: a tile is 256 x 256, each CTA has 128 of its rows, loads its own rows of A and HALF of the weight rows, and the even CTA issues
// tcgen05.mma.cta_group::2 for both, which reads either half from where it lies.  An SM takes in about 64 bytes a cycle: a 64-wide k-step of a 128 x 256 tile brings 48 KB
// (plain bf16) for 512 cycles of MMAs, 64 KB (two planes) for 1024; half of the weights' 32 KB comes off that here.
// One schedule over pairs ("cta" of TcSched); epilogue, parking and fix-up are each CTA's own, for its 128 rows: counters and partial tiles are per CTA.
// =====================================================================================
template <bool SPLIT>
struct Gemm2Cfg {
    static constexpr int BN = 256;
    static constexpr int A_BYTES = GEMM_BM * GEMM_BK * 2;
    static constexpr int B_BYTES = BN / 2 * GEMM_BK * 2;
    static constexpr int STAGE_BYTES = A_BYTES * (SPLIT ? 2 : 1) + B_BYTES;     // [A hi | A lo (SPLIT) | half of B]
    static constexpr int STAGES = GEMM_STAGE_BUDGET / STAGE_BYTES;
    static constexpr int EPI_BYTES = EPI_WARPS * EPI_PATCH;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_BYTES + 1024 /*align*/ + 256 /*barriers*/;
    static_assert((2 * STAGES + 4) * 8 + 12 <= 256, "barrier area");
};
template <int MODE, bool SPLIT>
__global__ void __launch_bounds__(512, 1) __cluster_dims__(2, 1, 1)
gemm_tc2_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmAlo, const __grid_constant__ CUtensorMap tmB,
                const __grid_constant__ CUtensorMap tmO, const __grid_constant__ CUtensorMap tmOlo, GemmEpi ep, int M, int N, int K, TcSched sc, int* err) {
    using Cfg = Gemm2Cfg<SPLIT>;
    constexpr int STAGES = Cfg::STAGES, BN = Cfg::BN;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* epi_smem = smem + STAGES * Cfg::STAGE_BYTES;
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(epi_smem + Cfg::EPI_BYTES);      // of the even CTA: both CTAs' operands of a stage
    uint64_t* empty_bar = full_bar + STAGES;           // of each CTA
    uint64_t* tmem_full_bar = empty_bar + STAGES;      // [2] of each CTA: accumulator b complete
    uint64_t* tmem_empty_bar = tmem_full_bar + 2;      // [2] of the even CTA: accumulator b drained by the epilogue warps of both
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty_bar + 2);
    int* last_flag = reinterpret_cast<int*>(tmem_slot + 1);
    int* gave_up = last_flag + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)cluster_rank(), pair = blockIdx.x >> 1;
    const TcWait wait{gave_up, err, peer_smem(gave_up, rank ^ 1)};
    const int KB = sc.KB;
    const int it_begin = sched_start(sc, pair), it_end = sched_start(sc, pair + 1);
    unsigned long long* prof = ep.prof ? ep.prof + 8 * (size_t)blockIdx.x : nullptr;       // (stamps 2 and 3, the MMAs': the even CTA's)
    auto stamp = [&](int i) {
        if (prof) { unsigned long long t; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t)); prof[i] = t; }
    };
    if (threadIdx.x == 0) stamp(0);

    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmA);
        if (SPLIT) tma_prefetch_desc(&tmAlo);
        tma_prefetch_desc(&tmB);
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full_bar[b], 1); mbar_init(&tmem_empty_bar[b], 2 * EPI_WARPS); }
        *gave_up = 0;
        fence_barrier_init();
    }
    if (warp == 2) { tmem_alloc_pair(tmem_slot, 2 * BN); tmem_relinquish_pair(); }
    tc_fence_before();
    __syncthreads();
    __syncwarp();
    cluster_sync_all();                             // the pair's barriers are initialised before either CTA signals the other's
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (threadIdx.x == 0) stamp(1);
    pdl_launch_dependents();
    if (warp == 0) {
        if (lane == 0) {
            constexpr int B_OFF = Cfg::A_BYTES * (SPLIT ? 2 : 1);
            const int npre = ep.w_dynamic ? 0 : min(it_end - it_begin, STAGES);
            int t = it_begin / KB, kb = it_begin - t * KB, mt, nt;
            sched_place(sc, pair, t, mt, nt);
            int n0 = nt * BN + rank * (BN / 2);
            for (int i = 0; i < npre; ++i) {        // the weights' first tiles go out before the dependency wait
                if (rank == 0) mbar_arrive_expect_tx(&full_bar[i], 2 * Cfg::STAGE_BYTES);
                tma_load_2d_pair(smem + i * Cfg::STAGE_BYTES + B_OFF, &tmB, peer_smem(&full_bar[i], 0), kb * GEMM_BK, n0);
                if (++kb == KB && i + 1 < npre) { kb = 0; sched_place(sc, pair, ++t, mt, nt); n0 = nt * BN + rank * (BN / 2); }
            }
            pdl_wait();
            int s = 0, left = npre; uint32_t ph = 0;
            for (int it = it_begin; it < it_end;) {
                t = it / KB;
                sched_place(sc, pair, t, mt, nt);
                const int seg_end = min(it_end, (t + 1) * KB), m0 = mt * (2 * GEMM_BM) + rank * GEMM_BM;
                n0 = nt * BN + rank * (BN / 2);
                int kc = (it - t * KB) * GEMM_BK;
                for (; it < seg_end; ++it, kc += GEMM_BK) {
                    uint8_t* a_dst = smem + s * Cfg::STAGE_BYTES;
                    const uint32_t bar = peer_smem(&full_bar[s], 0);
                    if (left > 0) --left;
                    else {
                        wait(&empty_bar[s], ph ^ 1);
                        if (rank == 0) mbar_arrive_expect_tx(&full_bar[s], 2 * Cfg::STAGE_BYTES);
                        tma_load_2d_pair(a_dst + B_OFF, &tmB, bar, kc, n0);
                    }
                    tma_load_2d_pair(a_dst, &tmA, bar, kc, m0);
                    if (SPLIT) tma_load_2d_pair(a_dst + Cfg::A_BYTES, &tmAlo, bar, kc, m0);
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            constexpr uint32_t idesc = make_idesc_bf16(2 * GEMM_BM, BN);
            int s = 0; uint32_t ph = 0;
            int seg = 0;
            for (int it = it_begin; it < it_end; ++seg) {
                const int seg_end = min(it_end, (it / KB + 1) * KB);
                const int b = seg & 1;
                wait(&tmem_empty_bar[b], ((seg >> 1) & 1) ^ 1);       // both epilogues have drained this accumulator (first two: free)
                tc_fence_after();
                const uint32_t acc = tmem_base + (uint32_t)(b * BN);
                for (int i = it; i < seg_end; ++i) {
                    wait(&full_bar[s], ph);
                    if (i == it_begin && lane == 0) stamp(2);
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(smem + s * Cfg::STAGE_BYTES);
                    const uint64_t adesc = make_smem_desc_sw128(a_addr);
                    const uint64_t aldesc = make_smem_desc_sw128(a_addr + Cfg::A_BYTES);
                    const uint64_t bdesc = make_smem_desc_sw128(a_addr + Cfg::A_BYTES * (SPLIT ? 2 : 1));
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < GEMM_BK / 16; ++k) {
                            umma_bf16_pair(acc, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc, (uint32_t)((i != it) | (k != 0)));
                            if (SPLIT) umma_bf16_pair(acc, aldesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc, 1u);
                        }
                        umma_commit_pair(&empty_bar[s]);
                        if (i == seg_end - 1) umma_commit_pair(&tmem_full_bar[b]);
                    }
                    __syncwarp();
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
                it = seg_end;
            }
            if (lane == 0) stamp(3);
        }
    } else if (warp >= 4) {
        if (threadIdx.x == 128) { tma_prefetch_desc(&tmO); tma_prefetch_desc(&tmOlo); }
        pdl_wait();
        const int q = warp & 3, part = (warp - 4) >> 2;
        EpiPatch patch{epi_smem + (warp - 4) * EPI_PATCH, false};
        gemm_epilogue<MODE, BN, 2>(ep, tmO, tmOlo, patch, smem + (warp - 4) * 4 * EPI_PATCH, M, N, sc, pair, rank, it_begin, it_end, tmem_base, tmem_full_bar, wait, last_flag, q, part, lane,
                                   [&] { stamp(4); }, [&](int b) { mbar_arrive_peer(peer_smem(&tmem_empty_bar[b], 0)); });
        if (lane == 0) tma_store_wait_read<0>();
        if (threadIdx.x == 128) stamp(5);
    }
    tc_fence_before();
    __syncthreads();
    __syncwarp();
    if (threadIdx.x == 0) stamp(6);
    cluster_sync_all();                             // neither CTA leaves while the other's MMAs read its operands or its warps signal here
    wait.drain();                                   // (a wait of either CTA ran out: copies and MMAs in flight reach into both)
    if (warp == 2) { tc_fence_after(); tmem_dealloc_pair(tmem_base, 2 * BN); if (lane == 0) stamp(7); }
}

// =====================================================================================
// SIMT debugging kernel (bring-up A/B for the tcgen05 path; never on the product path)
// =====================================================================================
template <int MODE>
__global__ void __launch_bounds__(128)
gemm_simt_kernel(const bf16* __restrict__ A, const bf16* __restrict__ A_lo, int lda, const bf16* __restrict__ W, GemmEpi ep, int M, int N, int K) {
    __shared__ float ws[32][65];
    const int m = blockIdx.y * 128 + threadIdx.x;
    const int n0 = blockIdx.x * 32;
    float acc[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) acc[j] = 0.f;
    for (int k0 = 0; k0 < K; k0 += 64) {
        __syncthreads();
        for (int i = threadIdx.x; i < 32 * 64; i += 128) {
            const int r = i >> 6, c = i & 63;
            ws[r][c] = (n0 + r < N) ? __bfloat162float(W[(size_t)(n0 + r) * K + k0 + c]) : 0.f;
        }
        __syncthreads();
        if (m < M) {
            for (int c = 0; c < 64; ++c) {
                float a = __bfloat162float(A[(size_t)m * lda + k0 + c]);
                if (A_lo != nullptr) a += __bfloat162float(A_lo[(size_t)m * lda + k0 + c]);
#pragma unroll
                for (int j = 0; j < 32; ++j) acc[j] = fmaf(a, ws[j][c], acc[j]);
            }
        }
    }
    if (m < M && n0 < N) {
        if (ep.bias != nullptr)
            for (int j = 0; j < 32; ++j) acc[j] += ep.bias[n0 + j];
        if (ep.col_scale != nullptr)
            for (int j = 0; j < 32; ++j) acc[j] *= ep.col_scale[n0 + j];
        if (ep.gate != nullptr)
            for (int j = 0; j < 32; ++j) acc[j] *= 1.f / (1.f + expf(-(ep.gate[(size_t)m * ep.ldg + n0 + j] + (ep.gate_bias ? ep.gate_bias[n0 + j] : 0.f))));
        epi_store32<MODE>(ep, m, n0, acc, true);
    }
}

// =====================================================================================
// Host side
// =====================================================================================
// CRANE_B200_GEMM_MINIT: fewest k-steps worth giving a CTA (below that the fixed cost of a CTA -- setup, first operand latency,
// parking and re-reading partial tiles -- outweighs the parallelism)
static const int g_gemm_minit = [] { const char* e = getenv("CRANE_B200_GEMM_MINIT"); const int v = e ? atoi(e) : 0; return v > 0 ? v : 8; }();

// Whole tiles are dealt in turn, eight rows of tiles wide: the CTAs at work at one time then read 8 strips of A and about 9 of the weights between them.  Each CTA a run of
// its own (one strip of the weights per CTA, all of A, 200 MB in use) read 5.0 GB for 24576 x 4096 at 4096 rows in split mode, 1174 us under the power limit; so 0.70 GB,
// 980 us.  Bands of 4 and of all 16 rows: within 1 % of that.  Tiles shared along K stay in runs: their order is part of the results.
static int sched_band(const TcSched& sc, bool stream_k) { return stream_k ? sc.tiles_m : std::min(8, sc.tiles_m); }

// maps of the results: patches of 32 rows (see epi_rows)
template <int MODE>
static bool out_maps(const GemmEpi& epi, int M, int N, CUtensorMap* tmO, CUtensorMap* tmOlo) {
    constexpr bool F32 = MODE == EPI_STORE_F32 || MODE == EPI_RESID_F32, GLU = MODE == EPI_SILU_MUL_BF16;
    const uint64_t out_cols = GLU ? N / 2 : N;
    const CUtensorMapDataType ot = F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    constexpr CUtensorMapSwizzle osw = GLU ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_64B;
    return tc_tmap(tmO, epi.out, ot, (uint64_t)M, out_cols, (uint64_t)epi.ldo, 32, F32 || GLU ? 16 : 32, osw) &&
           tc_tmap(tmOlo, !F32 && epi.out_lo ? epi.out_lo : epi.out, ot, (uint64_t)M, out_cols, (uint64_t)epi.ldo, 32, F32 || GLU ? 16 : 32, osw);
}

template <int BN, int MODE, bool SPLIT>
static int launch_tc(cudaStream_t stream, const bf16* A, const bf16* A_lo, int lda, const bf16* W, int M, int N, int K, const GemmEpi& epi,
                     bool stream_k) {
    using Cfg = GemmCfg<BN, SPLIT>;
    CUtensorMap tmA, tmAlo, tmB;
    if (!tc_tmap_bf16(&tmA, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, GEMM_BM)) return -1001;
    if (!tc_tmap_bf16(&tmAlo, SPLIT ? A_lo : A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, GEMM_BM)) return -1001;
    if (!tc_tmap_bf16(&tmB, W, (uint64_t)N, (uint64_t)K, (uint64_t)K, BN)) return -1001;
    CUtensorMap tmO, tmOlo;
    if (!out_maps<MODE>(epi, M, N, &tmO, &tmOlo)) return -1001;
    int* err = nullptr;
    if (const int e = tc_err_word(stream, &err)) return e;
    static SmemOptIn seen;
    if (const int e = ensure_dyn_smem(gemm_tc_kernel<BN, MODE, SPLIT>, (size_t)Cfg::SMEM_BYTES, seen)) return e;
    TcSched sc = {};
    sc.tiles_m = (M + GEMM_BM - 1) / GEMM_BM;
    sc.tiles_n = (N + BN - 1) / BN;
    sc.KB = K / GEMM_BK;
    const long long tiles = (long long)sc.tiles_m * sc.tiles_n, iters = tiles * sc.KB;
    if (iters > 0x7fffffffLL) return -1000;
    const int cap = std::min(tc_device_sms(), GEMM_MAX_CTAS);
    sc.unit = stream_k ? 1 : sc.KB;
    sc.band = sched_band(sc, stream_k);
    const long long units = iters / sc.unit;
    sc.G = (int)std::max<long long>(1, std::min<long long>(cap, stream_k ? iters / g_gemm_minit : tiles));
    sc.base = (int)(units / sc.G);
    sc.rem = (int)(units % sc.G);
    if (sc.unit != sc.KB) {                          // (whole tiles dealt out: none is shared)
        TcScratch scratch;
        if (const int e = tc_scratch_get(stream, (int)tiles, &scratch)) return e;
        sc.ws = scratch.ws;
        sc.counters = scratch.counters;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sc.G);
    cfg.blockDim = dim3(128 + 32 * EPI_WARPS);
    cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    int na = 0;
    if (prefill_pdl()) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    return (int)cudaLaunchKernelEx(&cfg, gemm_tc_kernel<BN, MODE, SPLIT>, tmA, tmAlo, tmB, tmO, tmOlo, epi, M, N, K, sc, err);
}

template <int MODE, bool SPLIT>
static int launch_tc2(cudaStream_t stream, const bf16* A, const bf16* A_lo, int lda, const bf16* W, int M, int N, int K, const GemmEpi& epi, bool stream_k) {
    using Cfg = Gemm2Cfg<SPLIT>;
    CUtensorMap tmA, tmAlo, tmB, tmO, tmOlo;
    if (!tc_tmap_bf16(&tmA, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, GEMM_BM)) return -1001;
    if (!tc_tmap_bf16(&tmAlo, SPLIT ? A_lo : A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, GEMM_BM)) return -1001;
    if (!tc_tmap_bf16(&tmB, W, (uint64_t)N, (uint64_t)K, (uint64_t)K, Cfg::BN / 2)) return -1001;
    if (!out_maps<MODE>(epi, M, N, &tmO, &tmOlo)) return -1001;
    int* err = nullptr;
    if (const int e = tc_err_word(stream, &err)) return e;
    static SmemOptIn seen;
    if (const int e = ensure_dyn_smem(gemm_tc2_kernel<MODE, SPLIT>, (size_t)Cfg::SMEM_BYTES, seen)) return e;
    TcSched sc = {};
    sc.tiles_m = (M + 2 * GEMM_BM - 1) / (2 * GEMM_BM);
    sc.tiles_n = (N + Cfg::BN - 1) / Cfg::BN;
    sc.KB = K / GEMM_BK;
    const long long tiles = (long long)sc.tiles_m * sc.tiles_n, iters = tiles * sc.KB;
    if (iters > 0x7fffffffLL) return -1000;
    const int cap = std::min(tc_max_clusters(2), GEMM_MAX_CTAS / 2);
    sc.unit = stream_k ? 1 : sc.KB;
    sc.band = sched_band(sc, stream_k);
    const long long units = iters / sc.unit;
    sc.G = (int)std::max<long long>(1, std::min<long long>(cap, stream_k ? iters / g_gemm_minit : tiles));
    sc.base = (int)(units / sc.G);
    sc.rem = (int)(units % sc.G);
    if (sc.unit != sc.KB) {
        TcScratch scratch;
        if (const int e = tc_scratch_get(stream, (int)tiles * 2, &scratch)) return e;
        sc.ws = scratch.ws;
        sc.counters = scratch.counters;
    }
    return launch_k(gemm_tc2_kernel<MODE, SPLIT>, dim3(2 * sc.G), dim3(128 + 32 * EPI_WARPS), Cfg::SMEM_BYTES, stream, prefill_pdl(), tmA, tmAlo, tmB, tmO, tmOlo, epi, M, N, K, sc, err);
}

// Tile width and schedule from a cost model fitted on B200 (microseconds; 42 shapes of 77 - 4096 rows, every width and schedule):
//   a k-step costs t_k: 64- and 128-wide tiles wait for their operands, 128 x 256 ones for shared memory, which MMAs read at 96 bytes a cycle while TMA writes
//   64 (two planes) or 96 (one) into it: 128 is the limit.  (Split, 256 wide, us a step: 0.565 - 0.57 with 24 - 64 tiles at once, 0.57 - 0.58 with 80 - 112, 0.615 with 128 and 144, 0.70
//   with 148, where the chip's power and the L2 begin to tell; hence 0.565, 0.60 above 96 and 0.66 with every SM busy.)
//   whole tiles: each CTA runs ceil(tiles / CTAs) tiles, the epilogue of all but the last hidden under the next tile's MMAs;
//   stream-K:    tiles x k-steps dealt evenly to all SMs, and the last of a tile's c contributors adding the others' parts.
// Tiles of pairs (256 x 256): a k-step 0.31 us plain and 0.62 split with few tiles, 0.36 and 0.63 with every SM busy on the scale that gives the single tiles 0.42 and 0.66, two or three
// us more of setup and hand-over.  Worth it where the operands are what takes the time; not where a gated or GELU tile's epilogue does (9 us), nor with rows that fill 256 badly.  Their
// stream-K pays above one wave too, while all operands stay in the L2 (CTAs at different k-steps share nothing of what they read): 4096 x 12288 at 2048 rows 187 us, whole tiles 141; 6144 x 4096 at
// 2500 rows, split, 161 and 178.
//   The constants were fitted to whole tiles in runs; since they are dealt in turn (sched_band) both sides' whole tiles are faster.  us of launches by themselves, the best single tiles /
//   the best pairs / as planned, plain: 24576 x 4096 at 200 rows 62 / 56 / 68, 300 64 / 76 / 64, 512 89 / 78 / 78, 1111 173 / 165 / 173, 1700 255 / 230 / 231, 4096 546 / 484 / 484
//   6144 x 4096 at 784 44.4 / 45.7 / 45.7, 1111 53 / 52 / 52, 4096 159 / 142 / 143     4096 x 12288 at 512 65 / 54 / 70, 784 78 / 74 / 74, 1111 81 / 131 / 82, 4096 313 / 279 / 279
//   12288 x 2048 at 784 46 / 44 / 44, 1111 48 / 55 / 48, 4096 149 / 135 / 135
//   split: 24576 x 4096 at 512 148 / 142 / 142, 784 234 / 263 / 234, 4096 967 / 923 / 925     6144 x 4096 at 784 66 / 73 / 73, 1111 82 / 87 / 95, 4096 263 / 263 / 263
//   4096 x 4096 at 4096 187 / 180 / 179     4096 x 12288 at 1700 239 / 260 / 260, 4096 538 / 528 / 528     8256 x 1024 at 4096 101 / 95 / 99     7168 x 1024 92 / 88 / 91
//   13 shapes of these models at 8 row counts from 200 to 4096, either precision: within 4 % of the best of six pinned plans in 184 of 208, at most 1.30 of it.
constexpr int GEMM_PAIR = 512;          // GemmPlan::bn: 256 x 256 tiles of two CTAs
struct GemmPlan { int bn; bool stream_k; double cost; };
static GemmPlan gemm_plan(int mode, int M, int N, int K, bool split, int sms) {
    static const int g_mode = [] { const char* e = getenv("CRANE_B200_GEMM_SCHED"); return e ? atoi(e) : 0; }();   // 1: whole tiles, 2: stream-K
    const int tm = (M + GEMM_BM - 1) / GEMM_BM, KB = K / GEMM_BK;
    const bool light = mode == EPI_STORE_F32 || mode == EPI_RESID_F32 || mode == EPI_STORE_BF16 || mode == EPI_RELU2_BF16;
    GemmPlan best{64, false, 1e30};
    for (int bn : {256, 128, 64}) {
        if (g_gemm_bn && bn != g_gemm_bn && !(g_gemm_bn == GEMM_PAIR && (M <= GEMM_BM || N < 256))) continue;
        if (!g_gemm_bn && bn > 64 && N < bn) continue;
        const long long tiles = (long long)tm * ((N + bn - 1) / bn);
        const long long per = (tiles + std::min<long long>(tiles, sms) - 1) / std::min<long long>(tiles, sms);
        const double tk = split ? (bn == 256 ? (per > 1 ? 0.66 : tiles > 96 ? 0.60 : 0.565) : bn == 128 ? 0.405 : 0.35)
                                : (bn == 256 ? (per > 1 ? 0.42 : 0.34) : bn == 128 ? 0.267 : 0.25);
        const double fixed = 3.7 + (light ? 2.7 : 5.5) * bn / 256.0;
        const double whole = fixed + (double)per * KB * tk;
        const double it = std::max((double)tiles * KB / sms, (double)g_gemm_minit);
        const double contrib = KB / it + 1.0;
        const double sk = fixed + it * (bn == 256 ? (split ? 0.66 : 0.42) : tk) + contrib * (bn == 256 ? 2.3 : bn == 128 ? 1.9 : 1.3);
        if (g_mode != 2 && whole < best.cost) best = GemmPlan{bn, false, whole};
        // stream-K only below one wave of whole tiles: above it the extra partial-tile traffic costs more than the idle SMs
        if (g_mode != 1 && (tiles < sms || g_mode == 2) && tiles * KB >= 2LL * sms && sk < best.cost) best = GemmPlan{bn, true, sk};
    }
    const int pairs = std::min(tc_max_clusters(2), sms / 2);
    if (pairs > 0 && M > GEMM_BM && N >= 256 && (!g_gemm_bn || g_gemm_bn == GEMM_PAIR)) {
        const long long tiles = (long long)((M + 255) / 256) * ((N + 255) / 256), per = (tiles + pairs - 1) / pairs;
        const double tk = split ? (per > 1 ? 0.63 : 0.62) : (per > 1 ? 0.36 : 0.31), fixed = light ? 8.9 : 13.2;
        if (light || KB * tk >= 9. || g_gemm_bn) {
            const double whole = fixed + (double)per * KB * tk;
            if (g_mode != 2 && whole < best.cost) best = GemmPlan{GEMM_PAIR, false, whole};
            const double it = std::max((double)tiles * KB / pairs, (double)g_gemm_minit);
            const double sk = fixed + 6. + it * (split ? 0.63 : 0.36) + (KB / it + 1.0) * 2.3;
            const double operands = 2. * K * ((double)N + (double)M * (split ? 2 : 1));
            if (g_mode != 1 && operands <= 126e6 && tiles * KB >= 2LL * pairs && sk < best.cost) best = GemmPlan{GEMM_PAIR, true, sk};
        }
    }
    return best;
}

template <int MODE>
static int launch_mode(cudaStream_t stream, const bf16* A, const bf16* A_lo, int lda, const bf16* W, int M, int N, int K,
                       const GemmEpi& epi, bool use_simt) {
    if (use_simt) {
        dim3 grid(N / 32, (M + 127) / 128);
        gemm_simt_kernel<MODE><<<grid, 128, 0, stream>>>(A, A_lo, lda, W, epi, M, N, K);
        return (int)cudaGetLastError();
    }
    const GemmPlan p = gemm_plan(MODE, M, N, K, A_lo != nullptr, std::min(tc_device_sms(), GEMM_MAX_CTAS));
    if (p.bn == GEMM_PAIR) return A_lo != nullptr ? launch_tc2<MODE, true>(stream, A, A_lo, lda, W, M, N, K, epi, p.stream_k) : launch_tc2<MODE, false>(stream, A, nullptr, lda, W, M, N, K, epi, p.stream_k);
    if (A_lo != nullptr) {
        switch (p.bn) {
            case 256: return launch_tc<256, MODE, true>(stream, A, A_lo, lda, W, M, N, K, epi, p.stream_k);
            case 128: return launch_tc<128, MODE, true>(stream, A, A_lo, lda, W, M, N, K, epi, p.stream_k);
            default:  return launch_tc<64, MODE, true>(stream, A, A_lo, lda, W, M, N, K, epi, p.stream_k);
        }
    }
    switch (p.bn) {
        case 256: return launch_tc<256, MODE, false>(stream, A, nullptr, lda, W, M, N, K, epi, p.stream_k);
        case 128: return launch_tc<128, MODE, false>(stream, A, nullptr, lda, W, M, N, K, epi, p.stream_k);
        default:  return launch_tc<64, MODE, false>(stream, A, nullptr, lda, W, M, N, K, epi, p.stream_k);
    }
}

int gemm_tiles(int mode, int M, int N, int K, bool split, bool* stream_k) {
    *stream_k = true;
    if (gemm_rows_pays(mode, split ? 2 : 1, M, N, K)) return 0;
    const GemmPlan p = gemm_plan(mode, M, N, K, split, std::min(tc_device_sms(), GEMM_MAX_CTAS));
    *stream_k = p.stream_k;
    return p.bn;
}

int gemm_bf16_launch(cudaStream_t stream, const bf16* A, const bf16* A_lo, int lda, const bf16* W, int M, int N, int K,
                     const GemmEpi& epi, bool use_simt) {
    if (M <= 0 || N <= 0 || K <= 0 || (K % GEMM_BK) != 0 || (N % 32) != 0 || (lda % 8) != 0) return -1000;
    const int P = A_lo ? 2 : 1;
    if (!use_simt && epi.prof == nullptr && gemm_rows_pays(epi.mode, P, M, N, K)) {       // the weights are the tile and the rows its columns
        const bf16* planes[3] = {A, A_lo, nullptr};
        return gemm_rows_launch(stream, planes, P, lda, W, M, N, K, epi, prefill_pdl());
    }
    switch (epi.mode) {
        case EPI_STORE_F32:      return launch_mode<EPI_STORE_F32>(stream, A, A_lo, lda, W, M, N, K, epi, use_simt);
        case EPI_STORE_BF16:     return launch_mode<EPI_STORE_BF16>(stream, A, A_lo, lda, W, M, N, K, epi, use_simt);
        case EPI_RESID_F32:      return launch_mode<EPI_RESID_F32>(stream, A, A_lo, lda, W, M, N, K, epi, use_simt);
        case EPI_SILU_MUL_BF16:  return launch_mode<EPI_SILU_MUL_BF16>(stream, A, A_lo, lda, W, M, N, K, epi, use_simt);
        case EPI_GELU_ERF_BF16:  return launch_mode<EPI_GELU_ERF_BF16>(stream, A, A_lo, lda, W, M, N, K, epi, use_simt);
        case EPI_GELU_TANH_BF16: return launch_mode<EPI_GELU_TANH_BF16>(stream, A, A_lo, lda, W, M, N, K, epi, use_simt);
        case EPI_RELU2_BF16:     return launch_mode<EPI_RELU2_BF16>(stream, A, A_lo, lda, W, M, N, K, epi, use_simt);
        default: return -1000;
    }
}

}  // namespace cb
