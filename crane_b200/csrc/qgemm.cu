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
// The weight rows are the MMA's M = 128 rows and the activation rows its N (16 .. 64; a tile of TM = 128 activation rows is two MMAs of 64), so a decode batch pays for the columns it
// has.
//
// The unpacked weights go from registers to TMEM, the MMA's A operand there: 128 f16 columns of a super-block are 128 lanes x 64 columns, a lane's row being the row that
// its thread unpacks.  Through shared memory (an f16 tile written by the unpacking warps, a proxy fence, read back by the MMAs) a super-block of 128 x 64 cost
// 1.3 us in Q4_K and 2.1 in Q6_K: 64 KB written and 64 read back at 128 bytes a cycle, and an MMA of up to 32 columns takes 40 cycles for its
// 4 KB of A, 20 with A in TMEM (64 columns: 48 and 32; 128 columns 64 either way).
//
// What bounds it: at few rows the quantised bytes (decode), at many the bytes of the activation codes, the MMAs and the instructions that turn nibbles into f16 (about
// 1.2 per weight).  Hence the split of a CTA into roles that overlap: one thread that brings raw blocks by TMA, eight warps that unpack
// them, one TMA producer for the activation codes, one MMA issuer, four or eight warps that
// read accumulators.  Stream-K over (128 x TM tile, super-block): every SM has the same number of super-blocks whatever the shape; partial
// tiles are added in contributor order by the last to arrive, so a result does not depend on who that was.
#include "quant.cuh"
#include "tc.cuh"

#include <cuda_fp16.h>

#include <algorithm>
#include <cstdlib>

namespace cb {

constexpr int QT_MAX_CTAS = 160;

// TM activation rows per tile.  128 (K-quants): two MMAs' halves of 64 rows, each with one of the two sets of accumulators, so that the weights are unpacked once for both.
template <int QT, int TM>
struct QCfg {
    static constexpr int NH = TM > 64 ? 2 : 1, NT = TM / NH;    // halves, columns per MMA
    static constexpr int SB = QT == QT_Q4_K ? 144 : QT == QT_Q6_K ? 224 : 272;
    static constexpr int PLANES = QT == QT_Q6_K ? 2 : 1;
    static constexpr int GROUPS = QT == QT_Q8_0 ? 8 : 1;        // accumulators per super-block
    static constexpr int DG = QT == QT_Q8_0 ? 128 / NT : 1;     // ... that change hands together
    static constexpr bool MINS = QT == QT_Q4_K;
    static constexpr int D_COLS = (MINS ? 2 : DG) * NT;         // TMEM: two such sets,
    static constexpr int UPS = QT == QT_Q6_K ? 2 : 1;           // then units of unpacked weights, this many to a super-block
    static constexpr int U_COLS = 128 * PLANES / UPS, NU = (512 - 2 * D_COLS) / U_COLS > 3 ? 3 : (512 - 2 * D_COLS) / U_COLS;
    static constexpr int DEQ_WARPS = 8, RR = 2;                 // warps that unpack, two to 32 rows; a warp's share of a super-block: RR x 64 elements
    static constexpr int RAW_BYTES = 128 * SB, RAW_REGS = QT == QT_Q4_K ? 1 + 2 * RR : QT == QT_Q6_K ? 2 + 2 * RR : 4 * RR;      // (16-byte pieces a thread reads per unit)
    static constexpr int NR = QT == QT_Q4_K ? (TM > 64 ? 3 : TM > 32 ? 5 : TM > 16 ? 6 : 8) : QT == QT_Q6_K ? (TM > 32 ? 5 : 6) : (TM > 32 ? 3 : 4);
    static constexpr int NB = QT == QT_Q6_K || TM != 64 ? 4 : 3;  // ring of codes: one unit of NT rows each
    static constexpr int B2_BYTES = MINS ? NT * 32 : 0, B_BYTES = NT * 512 / UPS, STG_BYTES = B_BYTES + B2_BYTES;
    static constexpr int A2_BYTES = MINS ? 128 * 32 : 0;        // [NU]
    // rings of scales, in super-blocks.  Who writes the scales of `it` has seen the MMAs of an older one done, so the accumulators two hand-overs before that have
    // been read.  Weights: in Q4_K it - NU (NU + 2 places); in Q6_K, written a unit ahead, the first half of it - 2 (4); in Q8_0, a super-block ahead, it - 3, of
    // which at 16 rows only the super-block before it - 3 is known to have been read (NU + 3).  Activations: it - NB / NH or it - NB / UPS.
    static constexpr int NS = (QT == QT_Q4_K && NU > 2) || (QT == QT_Q8_0 && TM == 16) ? 8 : 4, ND = NB + 2;
    static constexpr int SCW_BYTES = GROUPS * 128 * (MINS ? 8 : 4);
    static constexpr int DX_BYTES = GROUPS * TM * 4;
    static constexpr int EPI_WARPS = TM > 16 ? 8 : 4;          // (a division of the gated unit takes a lane 160 cycles, and nothing overlaps it: the columns are spread)
    static constexpr int ACC = TM / (EPI_WARPS / 4);            // columns per epilogue thread
    static constexpr int CH = ACC > 32 ? 8 : 16;                // ... read at once
    static constexpr int GATHER = TM > 64 ? 1 : TM > 32 ? 2 : TM > 16 ? 3 : 4;      // parts of a shared tile on their way at once, 16 columns each
    static constexpr int THREADS = (EPI_WARPS + DEQ_WARPS + 3) * 32;
    // offsets from a 1024-byte boundary; the swizzled tiles first
    static constexpr int STG_PITCH = (STG_BYTES + 1023) / 1024 * 1024;
    static constexpr int OFF_A2 = NB * STG_PITCH, OFF_RAW = OFF_A2 + NU * A2_BYTES, OFF_SCW = OFF_RAW + NR * RAW_BYTES, OFF_DX = OFF_SCW + NS * SCW_BYTES,
                         OFF_BAR = OFF_DX + ND * DX_BYTES, SMEM = OFF_BAR + 512 + 1024;
    static_assert(SMEM <= 227 * 1024, "rings do not fit");
    static_assert(NU >= 2 && 2 * D_COLS + NU * U_COLS <= 512, "TMEM");
    static_assert(NH == 1 || QT != QT_Q8_0, "two halves share the two sets");
    static_assert(OFF_A2 % 1024 == 0 && OFF_RAW % 128 == 0 && OFF_DX % 16 == 0 && OFF_BAR % 8 == 0, "alignment");
};

struct QGemmArgs {
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

// One CTA's share (`cta` of a.sc.G) of one linear
template <int QT, int TM>
__device__ __forceinline__ void qgemm_body(const CUtensorMap& tmW, const CUtensorMap& tmX, const CUtensorMap& tmS, const QGemmArgs& a, const int cta) {
    using C = QCfg<QT, TM>;
    constexpr int NT = C::NT, NH = C::NH;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(sm + C::OFF_BAR);
    uint64_t *raw_full = bars, *raw_empty = raw_full + C::NR, *a_full = raw_empty + C::NR, *a_empty = a_full + C::NU, *b_full = a_empty + C::NU, *b_empty = b_full + C::NB,
             *dx_full = b_empty + C::NB, *d_full = dx_full + C::ND, *d_empty = d_full + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(d_empty + 2);
    int* last_flag = reinterpret_cast<int*>(tmem_slot + 1);
    int* gave_up = last_flag + 1;
    static_assert((2 * C::NR + 2 * C::NU + 2 * C::NB + C::ND + 4) * 8 + 12 <= 512, "barrier area");
    const TcWait wait{gave_up, a.err};

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int W_DEQ = C::EPI_WARPS, W_TMA = W_DEQ + C::DEQ_WARPS, W_MMA = W_TMA + 1, W_RAW = W_MMA + 1;
    const int KB = a.sc.KB, it_begin = sched_start(a.sc, cta), it_end = sched_start(a.sc, cta + 1);

    if (threadIdx.x == 0) {
        *gave_up = 0;
        for (int i = 0; i < C::NR; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], C::DEQ_WARPS); }
        for (int i = 0; i < C::NU; ++i) { mbar_init(&a_full[i], C::DEQ_WARPS); mbar_init(&a_empty[i], 1); }
        for (int i = 0; i < C::NB; ++i) { mbar_init(&b_full[i], 1); mbar_init(&b_empty[i], 1); }
        for (int i = 0; i < C::ND; ++i) mbar_init(&dx_full[i], 1);
        for (int i = 0; i < 2; ++i) { mbar_init(&d_full[i], 1); mbar_init(&d_empty[i], C::EPI_WARPS / NH); }
        fence_barrier_init();
    }
    if (warp == W_MMA) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_launch_dependents();

    // ------------------------------------------------------------------------------------------------ raw weights: 128 rows of one block
    if (warp >= W_RAW) {           // (the weights do not depend on the kernel ahead: no dependency wait; rows behind the last one are zeros)
        if (lane == 0) {
            tma_prefetch_desc(&tmW);
            int rs = 0, kb = it_begin % KB, tile = it_begin / KB, n0 = tile / a.sc.tiles_m * 128; uint32_t ph = 0;
            for (int it = it_begin; it < it_end; ++it) {
                wait(&raw_empty[rs], ph ^ 1);
                mbar_arrive_expect_tx(&raw_full[rs], C::RAW_BYTES);
                tma_load_2d(sm + C::OFF_RAW + rs * C::RAW_BYTES, &tmW, &raw_full[rs], kb * (C::SB / 2), n0);
                if (++rs == C::NR) { rs = 0; ph ^= 1; }
                if (++kb == KB) { kb = 0; ++tile; n0 = tile / a.sc.tiles_m * 128; }
            }
            wait.drain();
        }
    // ------------------------------------------------------------------------------------------------ activation codes and their scales by TMA
    } else if (warp == W_TMA) {
        if (lane == 0) {
            tma_prefetch_desc(&tmX);
            pdl_wait();
            int st = 0, ds = 0, kb = it_begin % KB, tile = it_begin / KB, m0 = tile % a.sc.tiles_m * TM; uint32_t ph = 0;
            for (int it = it_begin; it < it_end; ++it) {
#pragma unroll 1
                for (int g = 0; g < C::UPS * NH; ++g) {       // units, and the halves of each
                    const int n = g / NH, m = m0 + g % NH * NT;
                    wait(&b_empty[st], ph ^ 1);
                    if (g == 0) {
                        mbar_arrive_expect_tx(&dx_full[ds], C::DX_BYTES);
#pragma unroll
                        for (int q = 0; q < C::GROUPS; ++q)
                            bulk_load(sm + C::OFF_DX + ds * C::DX_BYTES + q * TM * 4, a.dx + (size_t)(kb * C::GROUPS + q) * a.ldd + m0, TM * 4, &dx_full[ds]);
                        if (++ds == C::ND) ds = 0;
                    }
                    mbar_arrive_expect_tx(&b_full[st], C::STG_BYTES);
                    uint8_t* dst = sm + st * C::STG_PITCH;
#pragma unroll
                    for (int c = 0; c < 4 / C::UPS; ++c) tma_load_2d(dst + c * NT * 128, &tmX, &b_full[st], kb * 256 + (n * (4 / C::UPS) + c) * 64, m);
                    if (C::MINS) tma_load_2d(dst + C::B_BYTES, &tmS, &b_full[st], kb * 16, m);
                    if (++st == C::NB) { st = 0; ph ^= 1; }
                }
                if (++kb == KB) { kb = 0; ++tile; m0 = tile % a.sc.tiles_m * TM; }
            }
            wait.drain();
        }
    // ------------------------------------------------------------------------------------------------ MMA issuer (the whole warp runs the loop)
    } else if (warp == W_MMA) {
        constexpr uint32_t idesc = make_idesc_f16(128, NT);
        int st = 0, us = 0, ds = 0; uint32_t ph = 0, uph = 0, dph = 0;
        for (int it = it_begin; it < it_end; ++it) {
#pragma unroll 1
            for (int g = 0; g < C::UPS; ++g) {
                const uint32_t ta = tmem + (uint32_t)(2 * C::D_COLS + us * C::U_COLS);
                if constexpr (QT == QT_Q8_0) {
                    wait(&b_full[st], ph);
                    wait(&a_full[us], uph);
                    const uint64_t bd = make_smem_desc_sw128(smem_u32(sm + st * C::STG_PITCH));
#pragma unroll
                    for (int s = 0; s < C::GROUPS / C::DG; ++s) {
                        wait(&d_empty[ds], dph ^ 1);
                        tc_fence_after();
                        const uint32_t d = tmem + (uint32_t)(ds * C::D_COLS);
                        if (elect_one()) {
#pragma unroll
                            for (int j = 0; j < 2 * C::DG; ++j) {
                                const int k = 2 * C::DG * s + j;
                                umma_ts(d + (j >> 1) * NT, ta + 8 * k, bd + (uint64_t)((k >> 2) * NT * 8 + 2 * (k & 3)), idesc, (uint32_t)(j & 1));
                            }
                            umma_commit(&d_full[ds]);
                            if (s == C::GROUPS / C::DG - 1) { umma_commit(&a_empty[us]); umma_commit(&b_empty[st]); }
                        }
                        __syncwarp();
                        if (++ds == 2) { ds = 0; dph ^= 1; }
                    }
                    if (++st == C::NB) { st = 0; ph ^= 1; }
                } else {
#pragma unroll 1
                    for (int h = 0; h < NH; ++h) {
                        if (g == 0) wait(&d_empty[ds], dph ^ 1);
                        wait(&b_full[st], ph);
                        if (h == 0) wait(&a_full[us], uph);
                        tc_fence_after();
                        const uint32_t bb = smem_u32(sm + st * C::STG_PITCH);
                        const uint64_t bd = make_smem_desc_sw128(bb);
                        const uint32_t d = tmem + (uint32_t)(ds * C::D_COLS), acc0 = (uint32_t)(g != 0);
                        if (elect_one()) {
#pragma unroll
                            for (int k = 0; k < 16 / C::UPS; ++k) {
                                const uint64_t bw = bd + (uint64_t)((k >> 2) * NT * 8 + 2 * (k & 3));
                                umma_ts(d, ta + 8 * k, bw, idesc, k == 0 ? acc0 : 1u);
                                if (C::PLANES == 2) umma_ts(d, ta + C::U_COLS / 2 + 8 * k, bw, idesc, 1u);
                            }
                            if (C::MINS)
                                umma_bf16(d + NT, make_smem_desc_sw32(smem_u32(sm + C::OFF_A2 + us * C::A2_BYTES)), make_smem_desc_sw32(bb + C::B_BYTES), idesc, 0u);
                            if (h == NH - 1) umma_commit(&a_empty[us]);
                            umma_commit(&b_empty[st]);
                            if (g == C::UPS - 1) umma_commit(&d_full[ds]);
                        }
                        __syncwarp();
                        // one half: the sets take turns by super-block; two: each has its own
                        if (NH == 1) { if (g == C::UPS - 1 && ++ds == 2) { ds = 0; dph ^= 1; } }
                        else if (++ds == 2) { ds = 0; if (g == C::UPS - 1) dph ^= 1; }
                        if (++st == C::NB) { st = 0; ph ^= 1; }
                    }
                }
                if (++us == C::NU) { us = 0; uph ^= 1; }
            }
        }
    // ------------------------------------------------------------------------------------------------ weights: blocks -> f16 integers
    } else if (warp >= W_DEQ) {
        // A lane has a row, the two warps of its 32 rows a half of every super-block each (Q6_K: the low or the high nibbles of every unit).  The raw bytes of the next unit are read into
        // registers before this one's stores are waited for, so that only the instructions stand between two units.
        const int dw = warp - W_DEQ, part = dw >> 2, row = (dw & 3) * 32 + lane;
        constexpr int RR = C::RR;
        const uint32_t lanes = (uint32_t)((dw & 3) * 32) << 16;
        const int units = (it_end - it_begin) * C::UPS;
        int rs = 0, us = 0; uint32_t rph = 0, uph = 0;
        uint4 raw[C::RAW_REGS];
        uint32_t raw1 = 0;
        auto fetch = [&](int u) {               // unit u: raw blocks of slot rs -> registers
            const int n = C::UPS == 1 ? 0 : u % C::UPS;
            if (n == 0) wait(&raw_full[rs], rph);
            const uint8_t* sb = sm + C::OFF_RAW + rs * C::RAW_BYTES + row * C::SB;
            if constexpr (QT == QT_Q4_K) {
                raw[0] = *reinterpret_cast<const uint4*>(sb);
#pragma unroll
                for (int j = 0; j < 2 * RR; ++j) raw[1 + j] = *reinterpret_cast<const uint4*>(sb + 16 + 32 * RR * part + 16 * j);
            } else if constexpr (QT == QT_Q6_K) {       // half n of the block
#pragma unroll
                for (int e = 0; e < 2; ++e) raw[e] = *reinterpret_cast<const uint4*>(sb + 128 + 32 * n + 16 * e);
#pragma unroll
                for (int j = 0; j < 2 * RR; ++j) raw[2 + j] = *reinterpret_cast<const uint4*>(sb + 64 * n + 16 * j);
                raw1 = *reinterpret_cast<const uint32_t*>(sb + 192 + 8 * n + 4 * part);       // scales: byte 2 * quarter + (element / 16)
                if (n == 0 && part == 0)
                    reinterpret_cast<float*>(sm + C::OFF_SCW + ((it_begin + u / C::UPS) & (C::NS - 1)) * C::SCW_BYTES)[row] =
                        4.f * __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short*>(sb + 208)));
            } else {
#pragma unroll
                for (int j = 0; j < 4 * RR; ++j) raw[j] = *reinterpret_cast<const uint4*>(sb + 64 * RR * part + 16 * j);
                float* scw = reinterpret_cast<float*>(sm + C::OFF_SCW + ((it_begin + u) & (C::NS - 1)) * C::SCW_BYTES) + (2 * RR * part) * 128 + row;
#pragma unroll
                for (int rr = 0; rr < RR; ++rr) {
                    const uint32_t d = *reinterpret_cast<const uint32_t*>(sb + 256 + 4 * (RR * part + rr));
                    scw[256 * rr] = __half2float(__ushort_as_half((unsigned short)(d & 0xffffu)));
                    scw[256 * rr + 128] = __half2float(__ushort_as_half((unsigned short)(d >> 16)));
                }
            }
            if (n == C::UPS - 1) {
                __syncwarp();
                if (lane == 0) mbar_arrive(&raw_empty[rs]);
                if (++rs == C::NR) { rs = 0; rph ^= 1; }
            }
        };
        if (units > 0) fetch(0);
        for (int u = 0; u < units; ++u) {
            const uint32_t ta = tmem + lanes + (uint32_t)(2 * C::D_COLS + us * C::U_COLS);
            wait(&a_empty[us], uph ^ 1);
            tc_fence_after();
            if constexpr (QT == QT_Q4_K) {
                const uint4 hdr = raw[0];
#pragma unroll
                for (int rr = 0; rr < RR; ++rr) {          // 64 elements: sub-blocks 2 g (low nibbles) and 2 g + 1 (high); ggml get_scale_min_k4
                    const int g = RR * part + rr;
                    const uint32_t y = hdr.y >> (16 * (g & 1)), z = hdr.w >> (16 * (g & 1));
                    const uint32_t sa = g < 2 ? y & 63 : (z & 0xF) | (((y >> 6) & 3) << 4), sb2 = g < 2 ? (y >> 8) & 63 : ((z >> 8) & 0xF) | (((y >> 14) & 3) << 4);
                    const uint32_t s_lo = h2_int(sa), o_lo = h2_mul(s_lo, h2_const(0xE400)), t = h2_int(sb2), s_hi = h2_mul(t, h2_const(0x2C00)), o_hi = h2_mul(t, h2_const(0xD400));
                    const uint32_t ww[8] = {raw[1 + 2 * rr].x, raw[1 + 2 * rr].y, raw[1 + 2 * rr].z, raw[1 + 2 * rr].w, raw[2 + 2 * rr].x, raw[2 + 2 * rr].y, raw[2 + 2 * rr].z, raw[2 + 2 * rr].w};
                    uint32_t o[32];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {          // (1024 + q) * s - 1024 * s and (1024 + 16 q) * s / 16 - 64 * s: one rounding, exact
                        const uint32_t v = ww[i], v8 = v >> 8;
                        o[2 * i] = h2_fma((v & 0x000F000Fu) | 0x64006400u, s_lo, o_lo);
                        o[2 * i + 1] = h2_fma((v8 & 0x000F000Fu) | 0x64006400u, s_lo, o_lo);
                        o[16 + 2 * i] = h2_fma((v & 0x00F000F0u) | 0x64006400u, s_hi, o_hi);
                        o[16 + 2 * i + 1] = h2_fma((v8 & 0x00F000F0u) | 0x64006400u, s_hi, o_hi);
                    }
                    tmem_st32(ta + (uint32_t)g * 32, o);
                }
                if (part == 1) {                           // offsets m_0 .. m_7, 64 times them; d and dmin for the accumulators' readers
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
                    uint8_t* a2 = sm + C::OFF_A2 + us * C::A2_BYTES + row * 32;
                    const int sw = ((row >> 2) & 1) << 4;
                    *reinterpret_cast<uint4*>(a2 + sw) = make_uint4(m[0], m[1], m[2], m[3]);
                    *reinterpret_cast<uint4*>(a2 + (sw ^ 16)) = make_uint4(m64[0], m64[1], m64[2], m64[3]);
                    reinterpret_cast<float2*>(sm + C::OFF_SCW + ((it_begin + u) & (C::NS - 1)) * C::SCW_BYTES)[row] =
                        make_float2(__half2float(__ushort_as_half((unsigned short)(hdr.x & 0xffffu))), __half2float(__ushort_as_half((unsigned short)(hdr.x >> 16))));
                    fence_proxy_async();                   // (the offsets' tile is in shared memory)
                }
            } else if constexpr (QT == QT_Q6_K) {
                // part 0: low nibbles, quarters q1 | q2 of the block's half; 1: high nibbles, q3 | q4
                const uint32_t lmul = part ? h2_const(0x2400) : h2_const(0x3400), lofs = part ? h2_const(0xCC00) : h2_const(0xDC00);    // 1/64, 1/4; -16, -256
                const uint32_t lm = part ? 0x00F000F0u : 0x000F000Fu;
#pragma unroll
                for (int q = 0; q < RR; ++q) {             // elements [32 q, 32 q + 32) of the 64
                    uint32_t lo[16], hi[16];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {          // e: elements [16 e, 16 e + 16) of a quarter; high plane: (1024 + v - 1024 - 2) * 4 f
                        const uint32_t f = h2_byte(raw1 >> (16 * q + 8 * e)), ls = h2_mul(f, lmul), lo_o = h2_mul(f, lofs), hs = h2_mul(f, h2_const(0x4400));
                        const uint32_t wl[4] = {raw[2 + 2 * q + e].x, raw[2 + 2 * q + e].y, raw[2 + 2 * q + e].z, raw[2 + 2 * q + e].w};
                        const int sh = 4 * part + 2 * q;
                        const uint32_t wh[4] = {raw[e].x >> sh, raw[e].y >> sh, raw[e].z >> sh, raw[e].w >> sh};
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint32_t v = wl[i], v8 = v >> 8, w = wh[i], w8 = w >> 8;
                            lo[8 * e + 2 * i] = h2_fma((v & lm) | 0x64006400u, ls, lo_o);
                            lo[8 * e + 2 * i + 1] = h2_fma((v8 & lm) | 0x64006400u, ls, lo_o);
                            hi[8 * e + 2 * i] = h2_mul(h2_add((w & 0x00030003u) | 0x64006400u, h2_const(0xE402)), hs);
                            hi[8 * e + 2 * i + 1] = h2_mul(h2_add((w8 & 0x00030003u) | 0x64006400u, h2_const(0xE402)), hs);
                        }
                    }
                    tmem_st16(ta + (uint32_t)(32 * part + 16 * q), lo);
                    tmem_st16(ta + (uint32_t)(C::U_COLS / 2 + 32 * part + 16 * q), hi);
                }
            } else {
#pragma unroll
                for (int rr = 0; rr < RR; ++rr) {
                    uint32_t o[32];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint4 qv = raw[4 * rr + c];
                        const uint32_t ww[4] = {qv.x ^ 0x80808080u, qv.y ^ 0x80808080u, qv.z ^ 0x80808080u, qv.w ^ 0x80808080u};   // + 128: 0 .. 255
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            o[8 * c + 2 * i] = h2_add((ww[i] & 0x00FF00FFu) | 0x64006400u, h2_const(0xE480));
                            o[8 * c + 2 * i + 1] = h2_add(((ww[i] >> 8) & 0x00FF00FFu) | 0x64006400u, h2_const(0xE480));
                        }
                    }
                    tmem_st32(ta + (uint32_t)(RR * part + rr) * 32, o);
                }
            }
            if (u + 1 < units) fetch(u + 1);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&a_full[us]);
            if (++us == C::NU) { us = 0; uph ^= 1; }
        }
    // ------------------------------------------------------------------------------------------------ accumulators -> f32 sums -> epilogue
    } else {
        pdl_wait();
        const int q = warp & 3, col0 = (warp >> 2) * C::ACC, row = q * 32 + lane;
        constexpr size_t TILE_F = (size_t)128 * TM;
        int ds = NH == 2 ? warp >> 2 : 0, xs = 0; uint32_t dph = 0, xph = 0;
        for (int it = it_begin; it < it_end;) {
            const int seg_end = min(it_end, (it / KB + 1) * KB), t = it / KB;
            const int n0 = (t / a.sc.tiles_m) * 128, m0 = (t % a.sc.tiles_m) * TM;
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
                    const uint32_t d = tmem + (uint32_t)(ds * C::D_COLS + (g % C::DG) * NT + (NH == 2 ? 0 : col0)) + ((uint32_t)(q * 32) << 16);
#pragma unroll
                    for (int c = 0; c < C::ACC; c += C::CH) {
                        uint32_t r[C::CH], s[C::CH];
                        if constexpr (C::CH == 16) { tmem_ld16_async(d + c, r); if (C::MINS) tmem_ld16_async(d + NT + c, s); }
                        else { tmem_ld8_async(d + c, r); if (C::MINS) tmem_ld8_async(d + NT + c, s); }
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < C::CH; j += 4) {
                            const float4 x = *reinterpret_cast<const float4*>(dx + g * TM + c + j);
                            const float xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                            for (int e = 0; e < 4; e += 2) {         // two columns an instruction, each rounded as by itself
                                uint64_t v = f2_mul(f2(dw, dw), f2(__uint_as_float(r[j + e]), __uint_as_float(r[j + e + 1])));
                                if (C::MINS) v = f2_fma(f2(-dm, -dm), f2(__uint_as_float(s[j + e]), __uint_as_float(s[j + e + 1])), v);
                                f2_split(f2_fma(v, f2(xv[e], xv[e + 1]), f2(acc[c + j + e], acc[c + j + e + 1])), acc[c + j + e], acc[c + j + e + 1]);
                            }
                        }
                    }
                    if (g % C::DG == C::DG - 1) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&d_empty[ds]);
                        if (NH == 2) dph ^= 1;
                        else if (++ds == 2) { ds = 0; dph ^= 1; }
                    }
                }
                if (++xs == C::ND) { xs = 0; xph ^= 1; }
            }
            bool finish = sole;
            if (!sole) {      // park the partial tile (column by column: a warp's store is 128 contiguous bytes); the last contributor adds them in order
                float* mine = a.sc.ws + (size_t)(2 * cta + (head ? 0 : 1)) * TILE_F + (size_t)col0 * 128 + row;
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
                    auto part = [&](int cc) { return a.sc.ws + (size_t)(2 * cc + (sched_start(a.sc, cc) < t * KB ? 1 : 0)) * TILE_F + (size_t)col0 * 128 + row; };
#pragma unroll
                    for (int c = 0; c < C::ACC; c += 16) {
                        float sum[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j) sum[j] = 0.f;
#pragma unroll 1
                        for (int cc = c_first; cc <= c_last; cc += C::GATHER) {
                            float x[C::GATHER][16];
#pragma unroll
                            for (int r = 0; r < C::GATHER; ++r) {
                                const float* p = part(min(cc + r, c_last)) + c * 128;
#pragma unroll
                                for (int j = 0; j < 16; ++j) x[r][j] = __ldcg(p + j * 128);
                            }
#pragma unroll
                            for (int r = 0; r < C::GATHER; ++r)
                                if (cc + r <= c_last) {
#pragma unroll
                                    for (int j = 0; j < 16; ++j) sum[j] += x[r][j];
                                }
                        }
#pragma unroll
                        for (int j = 0; j < 16; ++j) acc[c + j] = sum[j];
                    }
                    if (threadIdx.x == 0) a.sc.counters[t] = 0;
                }
                named_bar_sync(1, C::EPI_WARPS * 32);              // last_flag is rewritten by the next segment
            }
            if (finish) {
                const int n = n0 + row, cols = min(C::ACC, a.M - m0 - col0);
                if (a.epi == GEMV_SILU_MUL) {                       // rows interleaved (gate_j, up_j): neighbouring lanes
                    // the even lane takes the even columns, the odd lane the odd ones
                    const int odd = lane & 1;
                    float* y = a.y + (size_t)(m0 + col0 + odd) * a.ldy + (n >> 1);
#pragma unroll
                    for (int j = 0; j < C::ACC; j += 2, y += 2 * a.ldy) {
                        const float other = __shfl_xor_sync(0xffffffffu, odd ? acc[j] : acc[j + 1], 1);
                        const float v = silu_f(odd ? other : acc[j]) * (odd ? acc[j + 1] : other);
                        if (n < a.N && j + odd < cols) *y = v;
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
    if (warp == W_MMA) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

template <int QT, int TM>
__global__ void __launch_bounds__(QCfg<QT, TM>::THREADS, 1)
qgemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmS, const __grid_constant__ QGemmArgs a) {
    qgemm_body<QT, TM>(tmW, tmX, tmS, a, blockIdx.x);
}

// Linears of the same rows side by side, each dealt out over its own CTAs as by itself: at width 4096 k and v of 32 rows are 64 CTAs each, 21 us one behind the other and 16
// together; at width 1024 q, k and v are one launch.
struct QJob { CUtensorMap w, x, s; QGemmArgs a; int qt, cta0; };
struct QJobs { QJob j[3]; int n; };
template <int TM>
__global__ void __launch_bounds__(QCfg<QT_Q4_K, TM>::THREADS, 1)
qgemm_jobs_kernel(const __grid_constant__ QJobs jobs) {
    int i = jobs.n - 1;
    while (i > 0 && (int)blockIdx.x < jobs.j[i].cta0) --i;
    const QJob& j = jobs.j[i];
    const int cta = blockIdx.x - j.cta0;
    if (j.qt == QT_Q4_K) qgemm_body<QT_Q4_K, TM>(j.w, j.x, j.s, j.a, cta);
    else if (j.qt == QT_Q6_K) qgemm_body<QT_Q6_K, TM>(j.w, j.x, j.s, j.a, cta);
    else qgemm_body<QT_Q8_0, TM>(j.w, j.x, j.s, j.a, cta);
}

// maps, arguments and division of work of one linear; workspace and counters come later
static int q_prepare(int qt, int TM, const unsigned char* w, const QRows& x, int M, int N, int K, int epi, float* y, int ldy, QJob* out) {
    const int half = q_sb_bytes(qt) / 2, NT = std::min(TM, 64);
    if (!tc_tmap_16(&out->w, w, (uint64_t)N, (uint64_t)K / 256 * half, (uint64_t)K / 256 * half, 128, half, CU_TENSOR_MAP_SWIZZLE_NONE)) return -1001;
    if (!tc_tmap_16(&out->x, x.codes, (uint64_t)M, (uint64_t)K, (uint64_t)K, NT, 64, CU_TENSOR_MAP_SWIZZLE_128B)) return -1001;
    if (!tc_tmap_16(&out->s, x.bsum, (uint64_t)M, (uint64_t)K / 16, (uint64_t)K / 16, NT, 16, CU_TENSOR_MAP_SWIZZLE_32B)) return -1001;
    QGemmArgs& a = out->a;
    a = {};
    a.M = M; a.N = N; a.K = K; a.epi = epi; a.y = y; a.ldy = ldy; a.dx = x.dx; a.ldd = x.ldd;
    TcSched& sc = a.sc;
    sc.tiles_m = (M + TM - 1) / TM; sc.tiles_n = (N + 127) / 128; sc.KB = K / 256;
    const long long tiles = (long long)sc.tiles_m * sc.tiles_n, iters = tiles * sc.KB;
    if (iters > 0x7fffffffLL) return -1000;
    sc.unit = 1;
    sc.G = (int)std::max<long long>(1, std::min<long long>(std::min(tc_device_sms(), QT_MAX_CTAS), iters / 2));     // two super-blocks pay for a CTA's setup
    sc.base = (int)(iters / sc.G); sc.rem = (int)(iters % sc.G);
    out->qt = qt; out->cta0 = 0;
    return 0;
}

template <int QT, int TM>
static int qgemm_launch_t(cudaStream_t st, const unsigned char* w, const QRows& x, int M, int N, int K, int epi, float* y, int ldy, bool pdl) {
    using C = QCfg<QT, TM>;
    QJob j;
    if (const int e = q_prepare(QT, TM, w, x, M, N, K, epi, y, ldy, &j)) return e;
    static SmemOptIn seen;
    if (const int e = ensure_dyn_smem(qgemm_kernel<QT, TM>, (size_t)C::SMEM, seen)) return e;
    TcScratch s;
    if (const int e = tc_scratch_get(st, j.a.sc.tiles_m * j.a.sc.tiles_n, &s)) return e;
    j.a.sc.ws = s.ws; j.a.sc.counters = s.counters; j.a.err = s.err;
    return launch_k(qgemm_kernel<QT, TM>, dim3(j.a.sc.G), dim3(C::THREADS), C::SMEM, st, pdl, j.w, j.x, j.s, j.a);
}

// Activation rows per tile.  Above 64, tiles of 64 or of 128 (K-quants), which unpack a block of weights half as often and read twice the accumulators behind one set of
// MMAs.  Estimated us of either: super-blocks on the busiest CTA and a constant, fitted to launches behind one another in prompts of 65 .. 512 rows at widths
// 1024, 2048 and 4096; 64 / 128 rows wide, where the wide form does better or nearly so:
//   Q4_K  12288 x 2048  384 rows 43.1 / 43.2, 512 53.6 / 55.7     24576 x 4096  128 rows 52.1 / 52.2, 192 70.3 / 91.3, 256 92.2 / 87.1, 384 129 / 118, 512 169 / 155
//   Q6_K  2048 x 6144   384 36.4 / 40.4, 512 46.1 / 49.3          4096 x 12288  192 65.1 / 76.3, 256 81.8 / 78.3, 384 115 / 101, 512 148 / 124
static float qgemm_estimate(int qt, int TM, int M, int N, int K) {
    const long long iters = (long long)((M + TM - 1) / TM) * ((N + 127) / 128) * (K / 256), G = std::max<long long>(1, std::min<long long>(tc_device_sms(), iters / 2));
    const float most = (float)((iters + G - 1) / G);
    if (qt == QT_Q4_K) return TM == 64 ? 1.0f * most + 9.f : 1.6f * most + 20.f;
    return TM == 64 ? 1.57f * most + 16.f : 2.18f * most + 32.f;
}
// CRANE_B200_QGEMM_ROWS=16|32|64|128 pins it (tests, sweeps; 128: K-quants only)
int qgemm_rows(int qt, int M, int N, int K) {
    static const int pin = [] { const char* e = getenv("CRANE_B200_QGEMM_ROWS"); return e ? atoi(e) : 0; }();
    if (pin) return pin;
    if (M <= 64) return M <= 16 ? 16 : M <= 32 ? 32 : 64;
    return qt != QT_Q8_0 && qgemm_estimate(qt, 128, M, N, K) < qgemm_estimate(qt, 64, M, N, K) ? 128 : 64;
}

template <int QT>
static int qgemm_launch_q(cudaStream_t st, const unsigned char* w, const QRows& x, int M, int N, int K, int epi, float* y, int ldy, bool pdl) {
    switch (qgemm_rows(QT, M, N, K)) {
        case 16: return qgemm_launch_t<QT, 16>(st, w, x, M, N, K, epi, y, ldy, pdl);
        case 32: return qgemm_launch_t<QT, 32>(st, w, x, M, N, K, epi, y, ldy, pdl);
        case 64: return qgemm_launch_t<QT, 64>(st, w, x, M, N, K, epi, y, ldy, pdl);
        default:
            if constexpr (QT != QT_Q8_0) return qgemm_launch_t<QT, 128>(st, w, x, M, N, K, epi, y, ldy, pdl);
            return -1000;
    }
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

template <int TM>
static int qgemm_jobs_launch_t(cudaStream_t st, QJobs& jobs, int ctas, int tiles, bool pdl) {
    constexpr size_t smem = std::max(QCfg<QT_Q4_K, TM>::SMEM, std::max(QCfg<QT_Q6_K, TM>::SMEM, QCfg<QT_Q8_0, TM>::SMEM));
    static SmemOptIn seen;
    if (const int e = ensure_dyn_smem(qgemm_jobs_kernel<TM>, smem, seen)) return e;
    TcScratch s;
    if (const int e = tc_scratch_get(st, tiles, &s)) return e;
    int t = 0;
    for (int i = 0; i < jobs.n; ++i) {        // partial tiles and counters of their own
        TcSched& sc = jobs.j[i].a.sc;
        sc.ws = s.ws + (size_t)2 * jobs.j[i].cta0 * 128 * TM; sc.counters = s.counters + t; jobs.j[i].a.err = s.err;
        t += sc.tiles_m * sc.tiles_n;
    }
    return launch_k(qgemm_jobs_kernel<TM>, dim3(ctas), dim3(QCfg<QT_Q4_K, TM>::THREADS), smem, st, pdl, jobs);
}

int qgemm_many_launch(cudaStream_t st, const QMany* m, int n, const QRows& x, int M, int K, bool pdl, int* launches) {
    *launches = 0;
    for (int i = 0; i < n;) {
        if (M <= 0 || m[i].N <= 0 || K <= 0 || (K % 256) != 0 || M > x.ldd) return -1000;
        const int TM = qgemm_rows(m[i].qt, M, m[i].N, K);
        QJobs jobs = {};
        int ctas = 0, tiles = 0, e = 0;
        while (TM <= 64 && i + jobs.n < n && jobs.n < 3 && qgemm_rows(m[i + jobs.n].qt, M, m[i + jobs.n].N, K) == TM) {
            const QMany& k = m[i + jobs.n];
            QJob& j = jobs.j[jobs.n];
            if ((e = q_prepare(k.qt, TM, k.w, x, M, k.N, K, GEMV_STORE, k.y, k.ldy, &j))) return e;
            if (ctas + j.a.sc.G > std::min(tc_device_sms(), QT_MAX_CTAS)) break;
            j.cta0 = ctas;
            ctas += j.a.sc.G; tiles += j.a.sc.tiles_m * j.a.sc.tiles_n;
            ++jobs.n;
        }
        if (jobs.n < 2) {
            if ((e = qgemm_launch(st, m[i].qt, m[i].w, x, M, m[i].N, K, GEMV_STORE, m[i].y, m[i].ldy, pdl))) return e;
            ++i;
        } else {
            e = TM == 16 ? qgemm_jobs_launch_t<16>(st, jobs, ctas, tiles, pdl) : TM == 32 ? qgemm_jobs_launch_t<32>(st, jobs, ctas, tiles, pdl) : qgemm_jobs_launch_t<64>(st, jobs, ctas, tiles, pdl);
            if (e) return e;
            i += jobs.n;
        }
        ++*launches;
    }
    return 0;
}

}  // namespace cb
