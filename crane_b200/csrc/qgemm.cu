// GGUF-quantised linears for many activation rows on the tensor cores: y[m, n] = epilogue(sum_k W[n, k] . xq[m, k]), with the integer dots of
// candle's CPU `QMatMul::forward` (crane-core/src/ops/linear.rs:23-48).
//
// Exactness.  Activations are int8 codes (xquant_kernel<true>), weights are small integers times block scales.  Both sides go through
// tcgen05.mma kind::f16 as f16 INTEGERS, so every product is exact and the f32 accumulator holds the block's integer sum, exactly
// while it stays under 2^24 (a block of one sign near the ends of its ranges can reach 3.1e7 in Q4_K and 1.3e8 quarters in Q6_K: there the accumulator
// rounds each of its 16 to 32 steps, some 1e-7 of the block):
//   Q4_K  A = sc_j * q (<= 63 * 15: 10 bits), one accumulator per 256-element super-block; a second one takes sum_j m_j * bsum_j, the offsets'
//         share, as a K = 16 product of [m_j | 64 m_j] and [bsum mod 64 | bsum div 64]
//   Q6_K  A = sc * (q - 32) needs 12 bits, so it is two f16 planes, sc * ql / 4 and 4 * sc * (qh - 2), accumulated into the same columns
//   Q8_0  A = q, one accumulator per 32-element block (both sides have a scale per 32)
// and the block scales are applied in f32 when the accumulator is read, once per block: acc += (d_w D - dmin_w D2) d_x.
//
// The weight rows are the MMA's M = 128 rows and the activation rows its N (NT = 16 .. 128), so a decode batch pays for the columns it has.
//
// What bounds it: at few rows the quantised bytes (decode), at many the MMAs and, nearly as much, the instructions that turn nibbles into
// f16 (about 1.2 per weight) and scale accumulators.  Hence the split of a CTA into roles that overlap: one or four warps that copy raw blocks into a
// ring, eight that unpack them into swizzled f16 tiles, one TMA producer for the activation codes, one MMA issuer, four or eight warps that
// read accumulators.  Stream-K over (128 x NT tile, super-block): every SM has the same number of super-blocks whatever the shape; partial
// tiles are added in contributor order by the last to arrive, so a result does not depend on who that was.
#include "quant.cuh"
#include "tc.cuh"

#include <cuda_fp16.h>

#include <algorithm>

namespace cb {

constexpr int QT_MAX_CTAS = 160;
constexpr int DEQ_WARPS = 8;

// What paces the issuing warp (measured on B200, one CTA): an MMA of up to 64 columns 40 - 47 cycles, 128 columns 64; a wait that succeeds at once
// 160 - 200; a commit 46.  So a stage carries eight MMAs, weights and activations arrive on ONE barrier and leave on one, and accumulators
// change hands once per super-block (Q8_0: per stage).  (Stages of four MMAs with barriers of their own for either operand cost 2.1 us per
// super-block whatever the copies and the unpacking did: 54 us for 4096 x 24576 at 8 rows.)
template <int QT, int NT>
struct QCfg {
    static constexpr int SB = QT == QT_Q4_K ? 144 : QT == QT_Q6_K ? 224 : 272;
    static constexpr int PLANES = QT == QT_Q6_K ? 2 : 1;
    static constexpr int CH64 = QT == QT_Q6_K ? 1 : 2;      // 64-wide tiles of each operand per stage
    static constexpr int SPS = 4 / CH64;                        // stages per super-block
    static constexpr int A_BYTES = 128 * 128 * PLANES * CH64, B_BYTES = NT * 128 * CH64, STG_BYTES = A_BYTES + B_BYTES;
    static constexpr int RAW_BYTES = 128 * SB;
    static constexpr int NSTG = QT == QT_Q4_K ? (NT > 64 ? 2 : 3) : QT == QT_Q6_K ? (NT > 64 ? 3 : 4) : 2;
    static constexpr int NR = QT == QT_Q4_K ? (NT > 64 ? 4 : NT > 32 ? 3 : NT > 16 ? 4 : 5) : QT == QT_Q6_K ? (NT > 16 ? 2 : 3) : 3;
    static constexpr int GROUPS = QT == QT_Q8_0 ? 8 : 1;        // accumulators per super-block
    static constexpr int DG = QT == QT_Q8_0 ? 2 * CH64 : 1;     // ... that change hands together
    static constexpr bool MINS = QT == QT_Q4_K;
    static constexpr int D_COLS = (MINS ? 2 : DG) * NT;         // two such sets
    static constexpr int TMEM_COLS = 2 * D_COLS <= 32 ? 32 : 2 * D_COLS <= 64 ? 64 : 2 * D_COLS <= 128 ? 128 : 2 * D_COLS <= 256 ? 256 : 512;
    static constexpr int NS = 4;                                // ring of scales (see the note at their writers)
    static constexpr int SCW_BYTES = GROUPS * 128 * (MINS ? 8 : 4);
    static constexpr int DX_BYTES = GROUPS * NT * 4;
    static constexpr int A2_BYTES = MINS ? 128 * 32 : 0, B2_BYTES = MINS ? NT * 32 : 0;
    static constexpr int EPI_WARPS = NT > 32 ? 8 : 4;
    static constexpr int ACC = NT / (EPI_WARPS / 4);            // columns per epilogue thread
    static constexpr int RAW_WARPS = NT > 32 ? 1 : 4;           // (few rows: bound by these copies; many: registers are dearer)
    static constexpr int THREADS = (EPI_WARPS + DEQ_WARPS + 2 + RAW_WARPS) * 32;
    // offsets from a 1024-byte boundary; the swizzled tiles first
    static constexpr int OFF_A2 = NSTG * STG_BYTES, OFF_B2 = OFF_A2 + 2 * A2_BYTES,
                         OFF_RAW = OFF_B2 + 2 * B2_BYTES, OFF_SCW = OFF_RAW + NR * RAW_BYTES, OFF_DX = OFF_SCW + NS * SCW_BYTES,
                         OFF_BAR = OFF_DX + NS * DX_BYTES, SMEM = OFF_BAR + 512 + 1024;
    static_assert(SMEM <= 227 * 1024, "tile rings do not fit");
    static_assert(STG_BYTES % 1024 == 0 && OFF_A2 % 1024 == 0 && OFF_RAW % 128 == 0 && OFF_DX % 16 == 0 && OFF_BAR % 8 == 0, "alignment");
};

struct QGemmArgs {
    const unsigned char* w;        // [N, K / 256] blocks
    int M, N, K, epi;              // activation rows, weight rows
    float* y; int ldy;             // [M, ldy] (GEMV_SILU_MUL: [M, N / 2])
    const float* dx;               // [GROUPS * K / 256][ldd] activation scales
    int ldd;
    TcSched sc;
    int* err;
};

__device__ __forceinline__ uint32_t h2_fma(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t h2_add(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t h2_mul(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__host__ __device__ constexpr uint32_t h2_const(uint32_t bits) { return bits | (bits << 16); }
// a small unsigned integer as a pair of f16: 0x6400 is 1024, one unit per mantissa bit
__device__ __forceinline__ uint32_t h2_int(uint32_t v) { return h2_add(v * 0x00010001u + 0x64006400u, h2_const(0xE400)); }
// ... a signed byte (v + 128 is unsigned)
__device__ __forceinline__ uint32_t h2_byte(uint32_t v) { return h2_add(((v ^ 0x80u) & 0xffu) * 0x00010001u + 0x64006400u, h2_const(0xE480)); }

template <int QT, int NT>
__global__ void __launch_bounds__(QCfg<QT, NT>::THREADS, 1)
qgemm_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmS, QGemmArgs a) {
    using C = QCfg<QT, NT>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(sm + C::OFF_BAR);
    uint64_t *raw_full = bars, *raw_empty = raw_full + C::NR, *full = raw_empty + C::NR, *empty = full + C::NSTG, *dx_full = empty + C::NSTG,
             *d_full = dx_full + C::NS, *d_empty = d_full + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(d_empty + 2);
    int* last_flag = reinterpret_cast<int*>(tmem_slot + 1);
    int* gave_up = last_flag + 1;
    static_assert((2 * C::NR + 2 * C::NSTG + C::NS + 4) * 8 + 12 <= 512, "barrier area");
    const TcWait wait{gave_up, a.err};

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int W_DEQ = C::EPI_WARPS, W_TMA = W_DEQ + DEQ_WARPS, W_MMA = W_TMA + 1, W_RAW = W_MMA + 1;
    const int KB = a.sc.KB, it_begin = sched_start(a.sc, blockIdx.x), it_end = sched_start(a.sc, blockIdx.x + 1);

    if (threadIdx.x == 0) {
        *gave_up = 0;
        for (int i = 0; i < C::NR; ++i) { mbar_init(&raw_full[i], C::RAW_WARPS * 32); mbar_init(&raw_empty[i], DEQ_WARPS); }
        for (int i = 0; i < C::NSTG; ++i) { mbar_init(&full[i], DEQ_WARPS / C::SPS + 1); mbar_init(&empty[i], 1); }
        for (int i = 0; i < C::NS; ++i) mbar_init(&dx_full[i], 1);
        for (int i = 0; i < 2; ++i) { mbar_init(&d_full[i], 1); mbar_init(&d_empty[i], C::EPI_WARPS); }
        fence_barrier_init();
    }
    if (warp == W_MMA) { tmem_alloc(tmem_slot, C::TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_launch_dependents();

    // ------------------------------------------------------------------------------------------------ raw weights: 16-byte asynchronous copies
    if (warp >= W_RAW) {           // (the weights do not depend on the kernel ahead: no dependency wait)
        // A thread's pieces sit at the same places of every super-block's 128 rows, and those of 32 rows repeat CPB pieces later: CPB offsets in registers and no
        // arithmetic beside the copies.  (Worked out per piece, a division by CPB and a 64-bit product each, the single warp of the wide tiles took
        // 2 us per super-block and paced the kernel: 24576 x 4096 at 64 rows Q4_K 51.5 us, 40.9 so; Q6_K at 512 rows 405 and 289.)
        // Q8_0 at up to 32 rows works them out all the same: its four warps have the time, and with 17 copies of 16 bytes at once the HBM took longer (24576 x 4096: 16
        // rows 53.6 us, 51.2 so; 32 rows 64.6 and 59.8; K-quants, of 9 and 14 pieces, 33.7 / 34.0 and 53.7 / 55.1).
        constexpr bool PER_PIECE = QT == QT_Q8_0 && C::RAW_WARPS > 1;
        const int t = threadIdx.x - W_RAW * 32;
        constexpr int CPB = C::SB / 16, T = C::RAW_WARPS * 32, GRP = 128 / T;
        const uint32_t row_bytes = (uint32_t)KB * C::SB;
        uint32_t off[CPB];
#pragma unroll
        for (int j = 0; j < CPB; ++j) { const uint32_t q = j * T + t, r = q / CPB; off[j] = r * row_bytes + (q - r * CPB) * 16; }
        int rs = 0, kb = it_begin % KB, n0 = it_begin / KB / a.sc.tiles_m * 128, tile = it_begin / KB; uint32_t rph = 0;
        for (int it = it_begin; it < it_end; ++it) {
            wait(&raw_empty[rs], rph ^ 1);
            const uint8_t* src = a.w + (size_t)n0 * row_bytes + (size_t)kb * C::SB;
            const uint32_t dst = smem_u32(sm + C::OFF_RAW + rs * C::RAW_BYTES) + t * 16;
            if (!PER_PIECE && n0 + 128 <= a.N) {
#pragma unroll
                for (int g = 0; g < GRP; ++g)
#pragma unroll
                    for (int j = 0; j < CPB; ++j)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (g * CPB + j) * (T * 16)), "l"(src + (size_t)g * T * row_bytes + off[j]) : "memory");
            } else {                                    // (the last tile: rows behind the last one are zeros)
#pragma unroll (PER_PIECE ? CPB * GRP : 1)
                for (int j = 0; j < CPB * GRP; ++j) {
                    const uint32_t q = j * T + t, r = q / CPB;
                    const bool in = n0 + (int)r < a.N;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + j * (T * 16)), "l"(src + (in ? (size_t)r * row_bytes + (q - r * CPB) * 16 : 0)), "r"(in ? 16 : 0) : "memory");
                }
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&raw_full[rs])) : "memory");
            if (++rs == C::NR) { rs = 0; rph ^= 1; }
            if constexpr (PER_PIECE) { kb = (it + 1) % KB; n0 = (it + 1) / KB / a.sc.tiles_m * 128; }
            else if (++kb == KB) { kb = 0; ++tile; n0 = tile / a.sc.tiles_m * 128; }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    // ------------------------------------------------------------------------------------------------ activation codes and their scales by TMA
    } else if (warp == W_TMA) {
        if (lane == 0) {
            tma_prefetch_desc(&tmX);
            pdl_wait();
            int st = 0, ds = 0, kb = it_begin % KB, tile = it_begin / KB, m0 = tile % a.sc.tiles_m * NT; uint32_t ph = 0;
            for (int it = it_begin; it < it_end; ++it) {
                // Slot ds of the scales was last read for super-block it - 4.  Its successor's data may go in once the first stage of `it` is free: a stage
                // at most two super-blocks back has been multiplied then, and the accumulators kept that one behind the readers of it - 4.
                for (int g = 0; g < C::SPS; ++g) {
                    wait(&empty[st], ph ^ 1);
                    if (g == 0) {
                        mbar_arrive_expect_tx(&dx_full[ds], C::DX_BYTES);
#pragma unroll
                        for (int q = 0; q < C::GROUPS; ++q)
                            bulk_load(sm + C::OFF_DX + ds * C::DX_BYTES + q * NT * 4, a.dx + (size_t)(kb * C::GROUPS + q) * a.ldd + m0, NT * 4, &dx_full[ds]);
                        if (++ds == C::NS) ds = 0;
                    }
                    const bool mins = C::MINS && g == C::SPS - 1;
                    mbar_arrive_expect_tx(&full[st], C::B_BYTES + (mins ? C::B2_BYTES : 0));
#pragma unroll
                    for (int c = 0; c < C::CH64; ++c)
                        tma_load_2d(sm + st * C::STG_BYTES + C::A_BYTES + c * NT * 128, &tmX, &full[st], kb * 256 + (g * C::CH64 + c) * 64, m0);
                    if (mins) tma_load_2d(sm + C::OFF_B2 + (it & 1) * C::B2_BYTES, &tmS, &full[st], kb * 16, m0);
                    if (++st == C::NSTG) { st = 0; ph ^= 1; }
                }
                if (++kb == KB) { kb = 0; ++tile; m0 = tile % a.sc.tiles_m * NT; }
            }
            wait.drain();
        }
    // ------------------------------------------------------------------------------------------------ MMA issuer (the whole warp runs the loop)
    } else if (warp == W_MMA) {
        constexpr uint32_t idesc = make_idesc_f16(128, NT);
        int st = 0, ds = 0; uint32_t ph = 0, dph = 0;
        for (int it = it_begin; it < it_end; ++it) {
            for (int g = 0; g < C::SPS; ++g) {
                if (QT == QT_Q8_0 || g == 0) { wait(&d_empty[ds], dph ^ 1); tc_fence_after(); }
                wait(&full[st], ph);
                tc_fence_after();
                const uint32_t aa = smem_u32(sm + st * C::STG_BYTES), d = tmem + (uint32_t)(ds * C::D_COLS);
                const uint64_t ad = make_smem_desc_sw128(aa), bd = make_smem_desc_sw128(aa + C::A_BYTES);
                if (elect_one()) {
#pragma unroll
                    for (int c = 0; c < C::CH64; ++c)
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const uint64_t aw = ad + (uint64_t)(c * C::PLANES * 1024 + 2 * k), bw = bd + (uint64_t)(c * NT * 8 + 2 * k);
                            if constexpr (QT == QT_Q8_0) umma_bf16(d + (2 * c + (k >> 1)) * NT, aw, bw, idesc, (uint32_t)(k & 1));
                            else umma_bf16(d, aw, bw, idesc, (uint32_t)((g | c | k) != 0));
                            if (C::PLANES == 2) umma_bf16(d, aw + 1024, bw, idesc, 1u);
                        }
                    if (C::MINS && g == C::SPS - 1)
                        umma_bf16(d + NT, make_smem_desc_sw32(smem_u32(sm + C::OFF_A2 + (it & 1) * C::A2_BYTES)),
                                  make_smem_desc_sw32(smem_u32(sm + C::OFF_B2 + (it & 1) * C::B2_BYTES)), idesc, 0u);
                    umma_commit(&empty[st]);
                    if (QT == QT_Q8_0 || g == C::SPS - 1) umma_commit(&d_full[ds]);
                }
                __syncwarp();
                if (++st == C::NSTG) { st = 0; ph ^= 1; }
                if (QT == QT_Q8_0 || g == C::SPS - 1) { if (++ds == 2) { ds = 0; dph ^= 1; } }
            }
        }
    // ------------------------------------------------------------------------------------------------ weights: blocks -> f16 integers
    } else if (warp >= W_DEQ) {
        // A warp always works on the same one of a super-block's stages, 64 rows of a 64-wide tile or 32 rows of two: 128 independent elements per lane
        // between one pair of waits and one proxy fence.
        const int dw = warp - W_DEQ, stage = dw % C::SPS, row0 = (dw / C::SPS) * (64 / C::CH64) + lane;
        int rs = 0; uint32_t rph = 0, seq = (uint32_t)stage;
        for (int it = it_begin; it < it_end; ++it, seq += C::SPS) {
            const uint32_t st = seq % C::NSTG, ph = (seq / C::NSTG) & 1;
            wait(&raw_full[rs], rph);
            // With as many places as a super-block has stages, a warp's next place cannot be two uses ahead of it (the MMAs take the stages in
            // order); with fewer it can, so there the warp follows every stage's place and a parity never stands for the wrong use.
            if constexpr (C::NSTG < C::SPS) {
                for (uint32_t u = seq - (uint32_t)stage; u < seq; ++u) wait(&empty[u % C::NSTG], ((u / C::NSTG) & 1) ^ 1);
            }
            wait(&empty[st], ph ^ 1);
            uint8_t* scw = sm + C::OFF_SCW + (it & (C::NS - 1)) * C::SCW_BYTES;
#pragma unroll
            for (int rr = 0; rr < 2; ++rr) {
                const int row = C::CH64 == 2 ? row0 : row0 + 32 * rr, g = C::CH64 == 2 ? 2 * stage + rr : stage;        // g: which 64 of the 256 elements
                uint8_t* A = sm + st * C::STG_BYTES + (C::CH64 == 2 ? rr * 16384 : 0);
                const uint8_t* sb = sm + C::OFF_RAW + rs * C::RAW_BYTES + row * C::SB;
                if constexpr (QT == QT_Q4_K) {
                    const uint4 hdr = *reinterpret_cast<const uint4*>(sb);
                    const uint4 w0 = *reinterpret_cast<const uint4*>(sb + 16 + 32 * g), w1 = *reinterpret_cast<const uint4*>(sb + 32 + 32 * g);
                    // scales of sub-blocks 2g (low nibbles) and 2g + 1 (high): ggml get_scale_min_k4
                    const int sh = 16 * (g & 1);
                    const uint32_t y = hdr.y >> sh, z = hdr.w >> sh;
                    const uint32_t sa = g < 2 ? y & 63 : (z & 0xF) | (((y >> 6) & 3) << 4), sb2 = g < 2 ? (y >> 8) & 63 : ((z >> 8) & 0xF) | (((y >> 14) & 3) << 4);
                    const uint32_t s_lo = h2_int(sa), o_lo = h2_mul(s_lo, h2_const(0xE400)), t = h2_int(sb2), s_hi = h2_mul(t, h2_const(0x2C00)), o_hi = h2_mul(t, h2_const(0xD400));
                    const uint32_t ww[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
                    for (int c = 0; c < 4; ++c) {          // (1024 + q) * s - 1024 * s and (1024 + 16 q) * s / 16 - 64 * s: one rounding, exact
                        uint32_t lo[4], hi[4];
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const uint32_t v = ww[2 * c + i], v8 = v >> 8;
                            lo[2 * i] = h2_fma((v & 0x000F000Fu) | 0x64006400u, s_lo, o_lo);
                            lo[2 * i + 1] = h2_fma((v8 & 0x000F000Fu) | 0x64006400u, s_lo, o_lo);
                            hi[2 * i] = h2_fma((v & 0x00F000F0u) | 0x64006400u, s_hi, o_hi);
                            hi[2 * i + 1] = h2_fma((v8 & 0x00F000F0u) | 0x64006400u, s_hi, o_hi);
                        }
                        *reinterpret_cast<uint4*>(A + sw128_off(row, c)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                        *reinterpret_cast<uint4*>(A + sw128_off(row, 4 + c)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                    }
                    if (g == 3) {                          // offsets m_0 .. m_7, 64 times them; d and dmin for the accumulators' readers
                        uint32_t m[4], m64[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            uint32_t mj[2];
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const int q = 2 * j + e, b = 8 * (q & 3);
                                mj[e] = q < 4 ? (hdr.z >> b) & 63 : ((hdr.w >> (b + 4)) & 0xF) | (((hdr.z >> (b + 6)) & 3) << 4);
                            }
                            m[j] = h2_add((mj[0] | (mj[1] << 16)) + 0x64006400u, h2_const(0xE400));
                            m64[j] = h2_mul(m[j], h2_const(0x5400));
                        }
                        uint8_t* a2 = sm + C::OFF_A2 + (it & 1) * C::A2_BYTES + row * 32;
                        const int sw = ((row >> 2) & 1) << 4;
                        *reinterpret_cast<uint4*>(a2 + sw) = make_uint4(m[0], m[1], m[2], m[3]);
                        *reinterpret_cast<uint4*>(a2 + (sw ^ 16)) = make_uint4(m64[0], m64[1], m64[2], m64[3]);
                        reinterpret_cast<float2*>(scw)[row] = make_float2(__half2float(__ushort_as_half((unsigned short)(hdr.x & 0xffffu))), __half2float(__ushort_as_half((unsigned short)(hdr.x >> 16))));
                    }
                } else if constexpr (QT == QT_Q6_K) {
                    const int h = g >> 1, p = g & 1;       // p = 0: low nibbles, quarters q1 | q2 of half h; p = 1: high nibbles, q3 | q4
                    if (g == 0) reinterpret_cast<float*>(scw)[row] = 4.f * __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short*>(sb + 208)));
                    const uint32_t sw = *reinterpret_cast<const uint32_t*>(sb + 192 + 8 * h + 4 * p);       // scales: byte 2 * quarter + (element / 16)
                    const uint32_t lmul = p ? h2_const(0x2400) : h2_const(0x3400), lofs = p ? h2_const(0xCC00) : h2_const(0xDC00);    // 1/64, 1/4; -16, -256
                    const uint32_t lm = p ? 0x00F000F0u : 0x000F000Fu;
#pragma unroll
                    for (int e = 0; e < 2; ++e) {          // e: elements [16 e, 16 e + 16) of a quarter
                        const uint4 qh = *reinterpret_cast<const uint4*>(sb + 128 + 32 * h + 16 * e);
                        const uint32_t wh[4] = {qh.x >> (4 * p), qh.y >> (4 * p), qh.z >> (4 * p), qh.w >> (4 * p)};
#pragma unroll
                        for (int q = 0; q < 2; ++q) {      // q: which of the two quarters, elements [32 q, 32 q + 32) of the step
                            const uint4 ql = *reinterpret_cast<const uint4*>(sb + 64 * h + 32 * q + 16 * e);
                            const uint32_t f = h2_byte(sw >> (16 * q + 8 * e)), ls = h2_mul(f, lmul), lo_o = h2_mul(f, lofs);
                            // high plane: two bits at 2 q (after the shift by 4 p): (1024 + 4^q v - 1024 - 2 * 4^q) * 4 f / 4^q
                            const uint32_t hm = q ? 0x000C000Cu : 0x00030003u, hsub = q ? h2_const(0xE408) : h2_const(0xE402), hs = q ? f : h2_mul(f, h2_const(0x4400));
                            const uint32_t wl[4] = {ql.x, ql.y, ql.z, ql.w};
                            uint32_t lo[8], hi[8];
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const uint32_t v = wl[i], v8 = v >> 8, u = wh[i], u8 = u >> 8;
                                lo[2 * i] = h2_fma((v & lm) | 0x64006400u, ls, lo_o);
                                lo[2 * i + 1] = h2_fma((v8 & lm) | 0x64006400u, ls, lo_o);
                                hi[2 * i] = h2_mul(h2_add((u & hm) | 0x64006400u, hsub), hs);
                                hi[2 * i + 1] = h2_mul(h2_add((u8 & hm) | 0x64006400u, hsub), hs);
                            }
#pragma unroll
                            for (int c = 0; c < 2; ++c) {
                                const uint32_t off = sw128_off(row, 4 * q + 2 * e + c);
                                *reinterpret_cast<uint4*>(A + off) = make_uint4(lo[4 * c], lo[4 * c + 1], lo[4 * c + 2], lo[4 * c + 3]);
                                *reinterpret_cast<uint4*>(A + 16384 + off) = make_uint4(hi[4 * c], hi[4 * c + 1], hi[4 * c + 2], hi[4 * c + 3]);
                            }
                        }
                    }
                } else {
                    const uint32_t d2 = *reinterpret_cast<const uint32_t*>(sb + 256 + 4 * g);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint4 qv = *reinterpret_cast<const uint4*>(sb + 64 * g + 16 * c);
                        const uint32_t ww[4] = {qv.x ^ 0x80808080u, qv.y ^ 0x80808080u, qv.z ^ 0x80808080u, qv.w ^ 0x80808080u};   // + 128: 0 .. 255
                        uint32_t o[8];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            o[2 * i] = h2_add((ww[i] & 0x00FF00FFu) | 0x64006400u, h2_const(0xE480));
                            o[2 * i + 1] = h2_add(((ww[i] >> 8) & 0x00FF00FFu) | 0x64006400u, h2_const(0xE480));
                        }
                        *reinterpret_cast<uint4*>(A + sw128_off(row, 2 * c)) = make_uint4(o[0], o[1], o[2], o[3]);
                        *reinterpret_cast<uint4*>(A + sw128_off(row, 2 * c + 1)) = make_uint4(o[4], o[5], o[6], o[7]);
                    }
                    reinterpret_cast<float*>(scw)[(2 * g) * 128 + row] = __half2float(__ushort_as_half((unsigned short)(d2 & 0xffffu)));
                    reinterpret_cast<float*>(scw)[(2 * g + 1) * 128 + row] = __half2float(__ushort_as_half((unsigned short)(d2 >> 16)));
                }
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) { mbar_arrive(&full[st]); mbar_arrive(&raw_empty[rs]); }
            if constexpr (C::NSTG < C::SPS) {
                for (uint32_t u = seq + 1; u % C::SPS != 0; ++u) wait(&empty[u % C::NSTG], ((u / C::NSTG) & 1) ^ 1);
            }
            if (++rs == C::NR) { rs = 0; rph ^= 1; }
        }
    // ------------------------------------------------------------------------------------------------ accumulators -> f32 sums -> epilogue
    } else {
        pdl_wait();
        const int q = warp & 3, col0 = (warp >> 2) * C::ACC, row = q * 32 + lane;
        constexpr size_t TILE_F = (size_t)128 * NT;
        constexpr int CH = NT > 64 ? 8 : 16;                        // columns per read: what the registers leave room for
        int ds = 0, xs = 0; uint32_t dph = 0, xph = 0;
        for (int it = it_begin; it < it_end;) {
            const int seg_end = min(it_end, (it / KB + 1) * KB), t = it / KB;
            const int n0 = (t / a.sc.tiles_m) * 128, m0 = (t % a.sc.tiles_m) * NT;
            const bool sole = it % KB == 0 && seg_end - it == KB, head = it == it_begin;
            float acc[C::ACC];
#pragma unroll
            for (int j = 0; j < C::ACC; ++j) acc[j] = 0.f;
            for (; it < seg_end; ++it) {
                const uint8_t* scw = sm + C::OFF_SCW + (it & (C::NS - 1)) * C::SCW_BYTES;
                wait(&dx_full[xs], xph);
                const float* dx = reinterpret_cast<const float*>(sm + C::OFF_DX + xs * C::DX_BYTES) + col0;
#pragma unroll 1
                for (int g = 0; g < C::GROUPS; ++g) {
                    if (g % C::DG == 0) { wait(&d_full[ds], dph); tc_fence_after(); }
                    float dw, dm = 0.f;
                    if constexpr (C::MINS) { const float2 s = reinterpret_cast<const float2*>(scw)[row]; dw = s.x; dm = s.y; }
                    else dw = reinterpret_cast<const float*>(scw)[g * 128 + row];
                    const uint32_t d = tmem + (uint32_t)(ds * C::D_COLS + (g % C::DG) * NT + col0) + ((uint32_t)(q * 32) << 16);
#pragma unroll
                    for (int c = 0; c < C::ACC; c += CH) {
                        uint32_t r[CH], s[CH];
                        if constexpr (CH == 16) { tmem_ld16_async(d + c, r); if (C::MINS) tmem_ld16_async(d + NT + c, s); }
                        else { tmem_ld8_async(d + c, r); if (C::MINS) tmem_ld8_async(d + NT + c, s); }
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < CH; j += 4) {
                            const float4 x = *reinterpret_cast<const float4*>(dx + g * NT + c + j);
                            const float xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                float v = dw * __uint_as_float(r[j + e]);
                                if (C::MINS) v = fmaf(-dm, __uint_as_float(s[j + e]), v);
                                acc[c + j + e] = fmaf(v, xv[e], acc[c + j + e]);
                            }
                        }
                    }
                    if (g % C::DG == C::DG - 1) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&d_empty[ds]);
                        if (++ds == 2) { ds = 0; dph ^= 1; }
                    }
                }
                if (++xs == C::NS) { xs = 0; xph ^= 1; }
            }
            bool finish = sole;
            if (!sole) {      // park the partial tile (column by column: a warp's store is 128 contiguous bytes); the last contributor adds them in order
                float* mine = a.sc.ws + (size_t)(2 * blockIdx.x + (head ? 0 : 1)) * TILE_F + (size_t)col0 * 128 + row;
#pragma unroll
                for (int j = 0; j < C::ACC; ++j) mine[j * 128] = acc[j];
                __threadfence();
                named_bar_sync(1, C::EPI_WARPS * 32);
                const int c_first = sched_owner(a.sc, t * KB), c_last = sched_owner(a.sc, t * KB + KB - 1);
                if (threadIdx.x == 0) *last_flag = atomicAdd(&a.sc.counters[t], 1) == c_last - c_first;
                named_bar_sync(1, C::EPI_WARPS * 32);
                finish = *last_flag != 0;
                if (finish) {
                    __threadfence();
#pragma unroll
                    for (int j = 0; j < C::ACC; ++j) acc[j] = 0.f;
                    for (int cc = c_first; cc <= c_last; ++cc) {
                        const float* p = a.sc.ws + (size_t)(2 * cc + (sched_start(a.sc, cc) < t * KB ? 1 : 0)) * TILE_F + (size_t)col0 * 128 + row;
#pragma unroll
                        for (int j = 0; j < C::ACC; ++j) {
                            acc[j] += __ldcg(p + j * 128);
                            if ((j & 15) == 15) asm volatile("" ::: "memory");     // 16 loads in flight, not all: registers
                        }
                    }
                    if (threadIdx.x == 0) a.sc.counters[t] = 0;
                }
                named_bar_sync(1, C::EPI_WARPS * 32);              // last_flag is rewritten by the next segment
            }
            if (finish) {
                const int n = n0 + row, cols = min(C::ACC, a.M - m0 - col0);
                if (a.epi == GEMV_SILU_MUL) {                       // rows interleaved (gate_j, up_j): neighbouring lanes
                    float* y = a.y + (size_t)(m0 + col0) * a.ldy + (n >> 1);
                    const bool mine = !(lane & 1) && n < a.N;
#pragma unroll
                    for (int j = 0; j < C::ACC; ++j, y += a.ldy) {
                        const float up = __shfl_xor_sync(0xffffffffu, acc[j], 1);
                        if (mine && j < cols) *y = silu_f(acc[j]) * up;
                    }
                } else if (n < a.N) {
                    float* y = a.y + (size_t)(m0 + col0) * a.ldy + n;
                    if (a.epi == GEMV_RESID) {
#pragma unroll
                        for (int c = 0; c < C::ACC; c += 8, y += (size_t)8 * a.ldy) {
                            float o[8];
#pragma unroll
                            for (int j = 0; j < 8; ++j) o[j] = c + j < cols ? y[(size_t)j * a.ldy] : 0.f;
#pragma unroll
                            for (int j = 0; j < 8; ++j) if (c + j < cols) y[(size_t)j * a.ldy] = o[j] + acc[c + j];
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < C::ACC; ++j, y += a.ldy) if (j < cols) *y = acc[j];
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == W_MMA) { tc_fence_after(); tmem_dealloc(tmem, C::TMEM_COLS); }
}

template <int QT, int NT>
static int qgemm_launch_t(cudaStream_t st, const unsigned char* w, const QRows& x, int M, int N, int K, int epi, float* y, int ldy, bool pdl) {
    using C = QCfg<QT, NT>;
    CUtensorMap tmX, tmS;
    if (!tc_tmap_16(&tmX, x.codes, (uint64_t)M, (uint64_t)K, (uint64_t)K, NT, 64, CU_TENSOR_MAP_SWIZZLE_128B)) return -1001;
    if (!tc_tmap_16(&tmS, x.bsum, (uint64_t)M, (uint64_t)K / 16, (uint64_t)K / 16, NT, 16, CU_TENSOR_MAP_SWIZZLE_32B)) return -1001;
    static SmemOptIn seen;
    if (const int e = ensure_dyn_smem(qgemm_kernel<QT, NT>, (size_t)C::SMEM, seen)) return e;
    QGemmArgs a = {};
    a.w = w; a.M = M; a.N = N; a.K = K; a.epi = epi; a.y = y; a.ldy = ldy; a.dx = x.dx; a.ldd = x.ldd;
    TcSched& sc = a.sc;
    sc.tiles_m = (M + NT - 1) / NT; sc.tiles_n = (N + 127) / 128; sc.KB = K / 256;
    const long long tiles = (long long)sc.tiles_m * sc.tiles_n, iters = tiles * sc.KB;
    if (iters > 0x7fffffffLL) return -1000;
    sc.unit = 1;
    sc.G = (int)std::max<long long>(1, std::min<long long>(std::min(tc_device_sms(), QT_MAX_CTAS), iters / 2));     // two super-blocks pay for a CTA's setup
    sc.base = (int)(iters / sc.G); sc.rem = (int)(iters % sc.G);
    TcScratch s;
    if (const int e = tc_scratch_get(st, (int)tiles, &s)) return e;
    sc.ws = s.ws; sc.counters = s.counters; a.err = s.err;
    return launch_k(qgemm_kernel<QT, NT>, dim3(sc.G), dim3(C::THREADS), C::SMEM, st, pdl, tmX, tmS, a);
}

// Above 32 rows: tiles of 64 activation rows, or of 128 (K-quants only), which unpack a block of weights half as often but have two stages for their operands
// instead of three and twice the partial tile to park and add for every CTA that shares one.  Estimated us of either: super-blocks on the busiest CTA,
// CTAs per tile, a constant; fitted to launches back to back, 8 linears x 13 row counts (33 .. 512) at widths 1024, 2048, 4096.
// us of a prompt through one layer of Q4_K_M, every linear 64 wide / 128 wide / as estimated: width 4096  65 rows 292 / 392 / 287, 128 301 / 402 / 297, 256 447 / 500 / 427,
// 384 611 / 601 / 561, 512 770 / 724 / 697; width 2048  256 242 / 321 / 234, 512 341 / 385 / 337; width 1024  512 220 / 280 / 221.
// Launches by themselves with cold caches and a rested chip, 64 / 128 wide, where the wide form does better:
//   Q4_K  6144 x 1024   128 rows 15.8 / 19.6, 512 26.5 / 28.9                       2048 x 2048   256 16.7 / 23.8, 512 21.0 / 29.1
//         12288 x 2048  256 40.3 / 41.2, 512 69.2 / 63.9                            24576 x 4096  65 67.1 / 61.0, 128 68.9 / 63.2, 193 124 / 108, 512 238 / 198
//   Q6_K  2048 x 6144   256 37.1 / 55.1, 512 58.7 / 60.6                            4096 x 12288  192 83.1 / 94.4, 256 105 / 95.5, 512 196 / 153
// (Q8_0 reads an accumulator per 32 elements; at width 4096 a layer took 475 us at 128 rows and 1224 at 512 with 64, 655 and 1328 with 128.)
static float qgemm_estimate(int qt, int nt, int M, int N, int K) {
    const long long iters = (long long)((M + nt - 1) / nt) * ((N + 127) / 128) * (K / 256), G = std::max<long long>(1, std::min<long long>(tc_device_sms(), iters / 2));
    const float most = (float)((iters + G - 1) / G), sharing = (float)(K / 256) * (float)G / (float)iters;
    if (qt == QT_Q4_K) return nt == 64 ? 1.32f * most + 0.39f * sharing + 7.1f : 2.34f * most + 1.5f * sharing + 12.9f;
    return nt == 64 ? 2.13f * most + 0.5f * sharing + 7.5f : 3.36f * most + 5.f * sharing + 14.f;
}

template <int QT>
static int qgemm_launch_q(cudaStream_t st, const unsigned char* w, const QRows& x, int M, int N, int K, int epi, float* y, int ldy, bool pdl) {
    if (M <= 16) return qgemm_launch_t<QT, 16>(st, w, x, M, N, K, epi, y, ldy, pdl);
    if (M <= 32) return qgemm_launch_t<QT, 32>(st, w, x, M, N, K, epi, y, ldy, pdl);
    if constexpr (QT != QT_Q8_0) {
        if (qgemm_estimate(QT, 128, M, N, K) < qgemm_estimate(QT, 64, M, N, K)) return qgemm_launch_t<QT, 128>(st, w, x, M, N, K, epi, y, ldy, pdl);
    }
    return qgemm_launch_t<QT, 64>(st, w, x, M, N, K, epi, y, ldy, pdl);
}

int qgemm_launch(cudaStream_t st, int qt, const unsigned char* w, const QRows& x, int M, int N, int K, int epi, float* y, int ldy, bool pdl) {
    if (M <= 0 || N <= 0 || K <= 0 || (K % 256) != 0 || (epi == GEMV_SILU_MUL && (N % 2) != 0) || M > x.ldd) return -1000;
    switch (qt) {
        case QT_Q4_K: return qgemm_launch_q<QT_Q4_K>(st, w, x, M, N, K, epi, y, ldy, pdl);
        case QT_Q6_K: return qgemm_launch_q<QT_Q6_K>(st, w, x, M, N, K, epi, y, ldy, pdl);
        case QT_Q8_0: return qgemm_launch_q<QT_Q8_0>(st, w, x, M, N, K, epi, y, ldy, pdl);
        default: return -1000;
    }
}

}  // namespace cb
