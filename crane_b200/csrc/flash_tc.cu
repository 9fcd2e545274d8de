// Flash attention forward on tcgen05 (prefill and vision tower): 128 query rows x one head per CTA, scores and output in TMEM.
//
// What bounds it: in split precision (hi + lo bf16 planes, three products kept of each) the MMAs -- per 128 keys at D = 128 24 of 128 columns for the scores
// and 24 for the output, 3.1 k cycles, 3.9 k measured: the scores' operands, both in shared memory, take its 128 bytes a cycle, and K / V come in beside them -- and, just
// below, the 128 KB of K / V planes a tile brings from L2 and the softmax's exponentials and conversions.  Probabilities replace the scores they come from (two buffers
// in turn, two planes in the 32 columns of 32 scores), so the softmax of a tile, one row per thread, runs under the output's MMAs of the tile before: it waits
// for them only where the output has to be rescaled.  With columns of their own the probabilities of a tile waited for every one of those MMAs: us a launch
// before / so, 4096 rows x 32 heads D = 128 split 357 / 338, 4096 x 8 heads D = 256 split 227 / 197, 784 rows x 16 heads D = 64 split 21.2 / 19.7, 1111 x 16
// D = 128 plain 21.5 / 19.2.  Short calls are bound by latencies and by code that comes out of a cold instruction cache, so the loops over a
// tile's columns are loops (77 rows behind 1 500 keys, 16 heads: 27.6 / 24.5).
// (A second softmax group on alternate tiles, with three buffers, gained nothing: 3.9 k of its 4.9 k cycles a tile were MMAs, and short calls got 3 % longer.)
// Tiles are 128 keys (64 at D = 256): 64-key tiles were bound by the hand-overs, 2.9 us each, 662 us for 4096 rows x 32 heads, D = 128, causal, split
// (mma.sync, flash.cuh: 1690).
//
// One TMA producer, one MMA issuer, four softmax / epilogue warps (TMEM lane = query row = thread).  K and V stream through ONE ring of slots in
// the order the MMAs take them -- K of tile i + 1 ahead of V of tile i -- so a slot is refilled as soon as its dozen MMAs are done, whatever
// the tile: K slots are [BN keys x 64 KC columns] per plane, V slots [R keys x all columns] per plane, read as an MN-major operand.
// P goes from registers to TMEM as the A operand of P V.  The output is rescaled only when a row's maximum has grown by more than 2^8
// since the last time (any reference works as long as sums and output share it).  Heads vary fastest and query tiles run from
// the last (longest) to the first, so the tail of a causal launch is short work.
#include "prefill.cuh"
#include "tc.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace cb {
namespace cg = cooperative_groups;

template <int D, bool SPLIT>
struct FtcCfg {
    static constexpr int P = SPLIT ? 2 : 1;
    static constexpr int BN = D > 128 ? 64 : 128;                   // keys per tile
    static constexpr int KC = P == 1 ? D / 64 : 1;                  // 64-wide column tiles per K slot
    static constexpr int SLOT = KC * P * BN * 128;
    static constexpr int R = SLOT / (D * 2 * P) < BN ? SLOT / (D * 2 * P) : BN;      // keys per V slot
    static constexpr int RB = R < 64 ? R : 64;                      // ... per copy (a page has 64)
    static constexpr int NKS = D / 64 / KC, NVS = BN / R;           // slots per tile
    static constexpr int Q_BYTES = P * 128 * D * 2;
    static constexpr int NSLOT = (208 * 1024 - Q_BYTES) / SLOT;
    static constexpr int SMEM = Q_BYTES + NSLOT * SLOT + 1024;
    static constexpr int C_S = D;                                   // TMEM columns: O [0, D), two buffers of BN that scores arrive in and probabilities replace
    static_assert(NVS * R == BN && R >= 16 && NSLOT >= 4 && C_S + 2 * BN <= 512, "");
};

// 2^x; results under 2^-126 are zero (the reference trails the running maximum by up to 8, so a row's largest probability is 1 .. 2^8)
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// MN-major operand, SWIZZLE_128B: 64 columns (128 B) x 8 keys per 1 KB atom; `lbo` bytes between 64-column groups, 1 KB between groups of 8 keys
__device__ __forceinline__ uint64_t make_smem_desc_mn128(uint32_t smem_addr, uint32_t lbo) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(lbo >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

struct FtcMaps { CUtensorMap k[2], v[2]; };

template <int D, bool SPLIT, bool CAUSAL, bool PAGED>
__global__ void __launch_bounds__(256, 1)
flash_tc_kernel(const __grid_constant__ FtcMaps maps, FlashArgs a, int ns, int* err) {
    using C = FtcCfg<D, SPLIT>;
    constexpr int P = C::P, BN = C::BN;
    const int head = blockIdx.x / ns, rank = blockIdx.x % ns, z = blockIdx.z, q0 = (CAUSAL ? gridDim.y - 1 - blockIdx.y : blockIdx.y) * 128;
    pdl_wait();                                       // (sequence bounds of a ragged batch come from the kernel ahead)
    pdl_launch_dependents();
    const int row0 = a.seq_start ? a.seq_start[z] : 0, S = a.seq_len ? a.seq_len[z] : a.S;
    if (q0 >= S) return;
    const int kv_off = CAUSAL ? (a.seq_kv_offset ? a.seq_kv_offset[z] : a.kv_offset) : 0;
    const int T = CAUSAL ? kv_off + S : S, kvh = head / (a.nh / a.nkv);
    const int* btab = (PAGED && a.seq_slot) ? a.block_table + (size_t)a.seq_slot[z] * a.bt_stride : a.block_table;
    const int n_tiles = CAUSAL ? (kv_off + min(q0 + 127, S - 1)) / BN + 1 : (T + BN - 1) / BN;
    // sliding window: the first query row of the tile reaches furthest back; the tiles of the kept first keys that the window does not reach come first
    const int t_first = (CAUSAL && a.window > 0) ? max(0, kv_off + q0 - a.window + 1) / BN : 0;
    const int keep = (CAUSAL && a.window > 0) ? a.keep_first : 0, n_keep = min((keep + BN - 1) / BN, t_first), n_all = n_keep + n_tiles - t_first;
    // a cluster of ns CTAs shares the keys of a query tile
    const int w0 = rank * n_all / ns, n_walk = (rank + 1) * n_all / ns - w0;
    auto tile_at = [&](int i) { i += w0; return i < n_keep ? i : t_first + i - n_keep; };

    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* ring = sm + C::Q_BYTES;
    __shared__ uint64_t full[C::NSLOT], empty[C::NSLOT], q_full, s_full[2], p_full[2], pv_done[4];
    __shared__ uint32_t tmem_slot;
    __shared__ int gave_up;
    const TcWait wait{&gave_up, err};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        gave_up = 0;
        for (int i = 0; i < C::NSLOT; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        mbar_init(&q_full, 4);
        for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 4); }
        for (int i = 0; i < 4; ++i) mbar_init(&pv_done[i], 1);
        fence_barrier_init();
    }
    if (warp == 2) { tmem_alloc(&tmem_slot, 512); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    // normalise and store columns c0, c0 + step .. (16 at a time) of query row r, whose output, reference and sum are given
    auto store = [&](int c0, int step, float m, float l, int r, auto&& fetch) {
        const int qrow = q0 + r;
        float inv = 1.f / l;
        if (a.sink) {        // the sink joins the denominator only: rescale to the larger of the reference and the sink
            const float s2 = a.sink[head] * 1.4426950408889634f, mn = fmaxf(m, s2), c = exp2f(m - mn);
            inv = c / (l * c + exp2f(s2 - mn));
        }
        inv *= a.out_mult;
        const bool in = qrow < S;
        const size_t orow = (size_t)(row0 + qrow);
        if (in && a.gate && a.gate_heads) inv *= 1.f / (1.f + __expf(-a.gate[orow * a.g_stride + head]));
        bf16* o = a.out + orow * a.o_stride + head * D;
        const float* gt = (a.gate && !a.gate_heads) ? a.gate + orow * a.g_stride + head * D : nullptr;
#pragma unroll 1
        for (int c = c0; c < D; c += step) {
            float w[16];
            fetch(c, w);
            if (in) {
                uint32_t hi[8], lo[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    float o0 = w[2 * j] * inv, o1 = w[2 * j + 1] * inv;
                    if (gt) {
                        const float2 g = *reinterpret_cast<const float2*>(gt + c + 2 * j);
                        o0 *= 1.f / (1.f + __expf(-g.x)); o1 *= 1.f / (1.f + __expf(-g.y));
                    }
                    split_bf16x2(o0, o1, hi[j], lo[j]);
                }
                *reinterpret_cast<uint4*>(o + c) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(o + c + 8) = make_uint4(hi[4], hi[5], hi[6], hi[7]);
                if (SPLIT) {
                    *reinterpret_cast<uint4*>(o + a.out_lo_off + c) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                    *reinterpret_cast<uint4*>(o + a.out_lo_off + c + 8) = make_uint4(lo[4], lo[5], lo[6], lo[7]);
                }
            }
        }
    };

    float m_row = -INFINITY, l_row = 0.f;              // softmax warps: a row's reference and sum, for the cluster's merge
    if (warp == 0) {
        if (lane == 0 && n_walk > 0) {
            int st = 0; uint32_t ph = 0;
            auto next = [&]() {
                wait(&empty[st], ph ^ 1);
                mbar_arrive_expect_tx(&full[st], C::SLOT);
            };
            auto step = [&]() { if (++st == C::NSLOT) { st = 0; ph ^= 1; } };
            // first rows of a tile's two halves of 64 keys; a page past the last one that holds a key is not looked up (its keys are masked)
            struct Rows { int y[2]; };
            const int last_page = (T - 1) / KV_PAGE;
            auto origin = [&](int tile) {
                Rows o;
#pragma unroll
                for (int h = 0; h < 2; ++h) o.y[h] = PAGED ? (btab[min(tile * (BN / 64) + h, last_page)] * a.nkv + kvh) * 64 : row0 + tile * BN + 64 * h;
                return o;
            };
            const int x0 = PAGED ? 0 : kvh * D;
            auto load_k = [&](const Rows& o) {
                for (int s = 0; s < C::NKS; ++s) {
                    next();
#pragma unroll
                    for (int kc = 0; kc < C::KC; ++kc)
#pragma unroll
                        for (int p = 0; p < P; ++p)
#pragma unroll
                            for (int h = 0; h < BN / 64; ++h)
                                tma_load_2d(ring + st * C::SLOT + (kc * P + p) * (BN * 128) + h * 8192, &maps.k[p], &full[st], x0 + (s * C::KC + kc) * 64, o.y[h]);
                    step();
                }
            };
            auto load_v = [&](const Rows& o) {
                for (int s = 0; s < C::NVS; ++s) {
                    next();
#pragma unroll
                    for (int p = 0; p < P; ++p)
#pragma unroll
                        for (int c = 0; c < D / 64; ++c)
#pragma unroll
                            for (int h = 0; h < C::R / C::RB; ++h) {
                                const int key = s * C::R + h * C::RB;
                                tma_load_2d(ring + st * C::SLOT + (p * (D / 64) + c) * (C::R * 128) + h * (C::RB * 128), &maps.v[p], &full[st], x0 + c * 64,
                                            (key >= 64 ? o.y[1] : o.y[0]) + (key & 63));
                            }
                    step();
                }
            };
            Rows cur = origin(tile_at(0)), nxt = cur;
            load_k(cur);
            if (n_walk > 1) nxt = origin(tile_at(1));
            for (int i = 0; i < n_walk; ++i) {
                Rows ahead = nxt;
                if (i + 2 < n_walk) ahead = origin(tile_at(i + 2));      // (its block-table look-up is in flight under the waits below)
                if (i + 1 < n_walk) load_k(nxt);
                load_v(cur);
                cur = nxt; nxt = ahead;
            }
            wait.drain();
        }
    } else if (warp == 1) {
        constexpr uint32_t id_s = make_idesc_bf16(128, BN), id_o = make_idesc_bf16(128, D) | (1u << 16);      // (B of P V: MN-major)
        const uint64_t qd = make_smem_desc_sw128(smem_u32(sm));
        int st = 0; uint32_t ph = 0;
        wait(&q_full, 0);
        auto scores = [&](int i) {
            const uint32_t d = tmem + C::C_S + (uint32_t)(i & 1) * BN;      // (the probabilities of tile i - 2 that were there: their MMAs are ahead of these)
            for (int s = 0; s < C::NKS; ++s) {
                wait(&full[st], ph);
                tc_fence_after();
                const uint64_t kd = make_smem_desc_sw128(smem_u32(ring + st * C::SLOT));
                if (elect_one()) {
#pragma unroll
                    for (int kc = 0; kc < C::KC; ++kc)
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const uint64_t qa = qd + (uint64_t)((s * C::KC + kc) * 1024 + 2 * k), kb = kd + (uint64_t)(kc * P * (BN * 8) + 2 * k);
                            constexpr uint64_t QLO = (uint64_t)(128 * D * 2) >> 4;
                            const uint32_t acc = (uint32_t)((s | kc | k) != 0);
                            if constexpr (SPLIT) {                     // small terms first
                                umma_bf16(d, qa + QLO, kb, id_s, acc);
                                umma_bf16(d, qa, kb + BN * 8, id_s, 1u);
                                umma_bf16(d, qa, kb, id_s, 1u);
                            } else umma_bf16(d, qa, kb, id_s, acc);
                        }
                    umma_commit(&empty[st]);
                    if (s == C::NKS - 1) umma_commit(&s_full[i & 1]);
                }
                __syncwarp();
                if (++st == C::NSLOT) { st = 0; ph ^= 1; }
            }
        };
        if (n_walk > 0) scores(0);
        for (int i = 0; i < n_walk; ++i) {
            if (i + 1 < n_walk) scores(i + 1);
            wait(&p_full[i & 1], (i >> 1) & 1);
            tc_fence_after();
            for (int s = 0; s < C::NVS; ++s) {
                wait(&full[st], ph);
                const uint32_t va = smem_u32(ring + st * C::SLOT);
                const uint64_t vd = make_smem_desc_mn128(va, C::R * 128), vl = make_smem_desc_mn128(va + (P - 1) * (C::SLOT / P), C::R * 128);
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < C::R / 16; ++k) {
                        const int key = s * C::R + k * 16;
                        const uint32_t pa = tmem + C::C_S + (uint32_t)((i & 1) * BN + (key >> 5) * 32 + ((key >> 4) & 1) * 8);
                        const uint32_t acc = (uint32_t)((i | s | k) != 0);
                        if constexpr (SPLIT) {
                            umma_ts(tmem, pa + 16, vd + (uint64_t)(k * 128), id_o, acc);
                            umma_ts(tmem, pa, vl + (uint64_t)(k * 128), id_o, 1u);
                            umma_ts(tmem, pa, vd + (uint64_t)(k * 128), id_o, 1u);
                        } else umma_ts(tmem, pa, vd + (uint64_t)(k * 128), id_o, acc);
                    }
                    umma_commit(&empty[st]);
                    if (s == C::NVS - 1) umma_commit(&pv_done[i & 3]);
                }
                __syncwarp();
                if (++st == C::NSLOT) { st = 0; ph ^= 1; }
            }
        }
    } else if (warp >= 4) {
        const int q = warp & 3, r = q * 32 + lane, qrow = q0 + r, qpos = kv_off + qrow;
        const uint32_t lanes = (uint32_t)(q * 32) << 16;
        // ---- the Q tile: swizzled [128 rows x 64 columns] tiles per plane, rows past S zero; asynchronous, so all of a warp's rows are in flight together ----
        for (int rr = q * 32; rr < q * 32 + 32; ++rr) {
            const bool in = q0 + rr < S;
            const bf16* src = a.q + (size_t)(row0 + min(q0 + rr, S - 1)) * a.q_stride + head * D;
#pragma unroll
            for (int e = lane; e < P * (D / 8); e += 32) {
                const int p = e / (D / 8), ch = e % (D / 8);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(sm + p * (128 * D * 2) + (ch >> 3) * 16384) + sw128_off(rr, ch & 7)),
                             "l"(src + (p ? a.q_lo_off : 0) + ch * 8), "r"(in ? 16 : 0) : "memory");
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&q_full);

        const float sl2 = a.scale * 1.4426950408889634f;
        const bool mods = (CAUSAL && (a.softcap > 0.f || a.dist_r1 || a.dist_table)) || !(sl2 > 0.f);
        const float mul = mods ? 1.f : sl2;           // exponent = mul * s - reference: the scale rides on the subtraction unless it was applied before
        const float inv_cap = a.softcap > 0.f ? 1.f / a.softcap : 0.f;
        const float dr1 = (CAUSAL && a.dist_r1) ? a.dist_r1[head] : 0.f, dr2 = (CAUSAL && a.dist_r1) ? a.dist_r2[head] : 0.f;
        const float* dtab = (CAUSAL && a.dist_table) ? a.dist_table + (size_t)head * a.dist_rows : nullptr;
        float m = -INFINITY, l = 0.f;                 // reference of the exponentials (not always the running maximum), sum
        for (int i = 0; i < n_walk; ++i) {
            const int kv0 = tile_at(i) * BN;
            wait(&s_full[i & 1], (i >> 1) & 1);
            tc_fence_after();
            const uint32_t sa = tmem + lanes + C::C_S + (uint32_t)(i & 1) * BN;
            if (mods) {                 // cap, then the distance terms, in f32 on the scaled score, in place (one copy of this code for 16 columns: unrolled over
#pragma unroll 1                        // the tile it outgrew the instruction cache and a tile took 64 k cycles)
                for (int c = 0; c < BN; c += 16) {
                    uint32_t w[16];
                    tmem_ld16_async(sa + c, w);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const int dist = max(0, qpos - (kv0 + c + j));
                        float sc = __uint_as_float(w[j]) * a.scale;
                        if (CAUSAL && a.softcap > 0.f) {            // tanh(x) = 1 - 2 / (e^{2x} + 1)
                            const float t = __expf(fminf(2.f * sc * inv_cap, 40.f));
                            sc = a.softcap * (1.f - __fdividef(2.f, t + 1.f));
                        }
                        if (CAUSAL && a.dist_r1) sc -= dr1 * log1pf(dr2 * (float)dist);
                        if (dtab) sc += dtab[min(dist, a.dist_rows - 1)];
                        w[j] = __float_as_uint(sc * 1.4426950408889634f);
                    }
                    tmem_st16(sa + c, w);
                }
                tmem_st_wait();
            }
            // every key of the tile visible to every row of this warp?  (the warp's first row sees the fewest new keys, its last the fewest old ones)
            const bool whole = kv0 + BN <= T && (!CAUSAL || (kv0 + BN - 1 <= kv_off + q0 + q * 32 && (a.window <= 0 || kv_off + q0 + q * 32 + 31 - kv0 < a.window)));
            if (!whole) {               // the row sees columns [lo, hi) of the tile and those below kp (in place, for the code's size)
                const int hi = (CAUSAL ? min(T, qpos + 1) : T) - kv0, lo = (CAUSAL && a.window > 0) ? qpos - a.window + 1 - kv0 : -1, kp = keep - kv0;
#pragma unroll 1
                for (int c = 0; c < BN; c += 16) {
                    uint32_t w[16];
                    tmem_ld16_async(sa + c, w);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) if (!(c + j < hi && (c + j >= lo || c + j < kp))) w[j] = 0xff800000u;
                    tmem_st16(sa + c, w);
                }
                tmem_st_wait();
            }
            // Both passes over the scores are loops over 64 columns that read them from TMEM: code that a CTA with two or three tiles runs once or twice comes out of a cold
            // instruction cache (unrolled over 128 columns, its first exponentials took 6 k cycles and the next tile's 2.2 k).
            constexpr int CH = 64;
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};      // (four chains: a warp has its scheduler to itself)
#pragma unroll 1
            for (int c0 = 0; c0 < BN; c0 += CH) {
                uint32_t u[CH];
#pragma unroll
                for (int c = 0; c < CH; c += 16) tmem_ld16_async(sa + c0 + c, u + c);
                tmem_ld_wait();
#pragma unroll
                for (int c = 0; c < CH; ++c) mx4[c & 3] = fmaxf(mx4[c & 3], __uint_as_float(u[c]));
            }
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * mul;
            const bool grow = mx > m + 8.f || (m == -INFINITY && mx > -INFINITY);
            if (__any_sync(0xffffffffu, grow)) {
                const float mn = fmaxf(m, mx), f = m == -INFINITY ? 0.f : exp2f(m - mn);
                l *= f;
                m = mn;
                if (i > 0) {
                    // O is whole.  (Four barriers in turn: when the scores of tile i are there, the MMAs of tile i - 2 are done, so a parity cannot stand for an older use.)
                    wait(&pv_done[(i - 1) & 3], ((i - 1) >> 2) & 1);
                    tc_fence_after();
#pragma unroll 1
                    for (int c = 0; c < D; c += 16) {
                        uint32_t o[16];
                        tmem_ld16_async(tmem + lanes + c, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * f);
                        tmem_st16(tmem + lanes + c, o);
                    }
                }
            }
            const float ref = m == -INFINITY ? 0.f : m;
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
            for (int c0 = 0; c0 < BN; c0 += CH) {
                uint32_t u[CH];
#pragma unroll
                for (int c = 0; c < CH; c += 16) tmem_ld16_async(sa + c0 + c, u + c);
                tmem_ld_wait();
                const float* s = reinterpret_cast<const float*>(u);
#pragma unroll
                for (int c = 0; c < CH; c += 32) {
                    uint32_t hi[16], lo[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float p0 = ex2(fmaf(s[c + 2 * j], mul, -ref)), p1 = ex2(fmaf(s[c + 2 * j + 1], mul, -ref));
                        sum[(2 * j) & 3] += p0; sum[(2 * j + 1) & 3] += p1;
                        split_bf16x2(p0, p1, hi[j], lo[j]);
                    }
                    tmem_st16(sa + c0 + c, hi);                           // in place of the 32 scores: 16 columns of either plane
                    if (SPLIT) tmem_st16(sa + c0 + c + 16, lo);
                }
            }
            l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
            tmem_st_wait();
            tc_fence_before();
            if (kv0 + BN > T) {       // the rows behind the last key are a page's never written rest or the next sequence's: zero times whatever is there must stay zero
                const int seq = n_walk * C::NKS + (n_walk - 1) * C::NVS;
                if (i > 0) wait(&pv_done[(i - 1) & 3], ((i - 1) >> 2) & 1);      // (every slot's use before its last has been filled: the parities below cannot stand for an older one)
                for (int j = 0; j < C::NVS; ++j) {
                    const int slot = (seq + j) % C::NSLOT, lo_r = max(0, T - kv0 - j * C::R);
                    if (lo_r >= C::R) continue;
                    wait(&full[slot], ((seq + j) / C::NSLOT) & 1);
                    const int per = (C::R - lo_r) * 8;          // 16-byte pieces per tile
                    for (int e = threadIdx.x - 128; e < P * (D / 64) * per; e += 128)
                        *reinterpret_cast<uint4*>(ring + slot * C::SLOT + (e / per) * (C::R * 128) + lo_r * 128 + (e % per) * 16) = make_uint4(0, 0, 0, 0);
                }
                fence_proxy_async();
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[i & 1]);
        }
        if (n_walk > 0) { wait(&pv_done[(n_walk - 1) & 3], ((n_walk - 1) >> 2) & 1); tc_fence_after(); }
        m_row = m; l_row = l;
        if (ns == 1) store(0, 16, m, l, r, [&](int c, float* v) {
            uint32_t* w = reinterpret_cast<uint32_t*>(v);
            tmem_ld16_async(tmem + lanes + c, w);
            tmem_ld_wait();
        });
    }
    if (ns > 1) {
        // CTA k merges and stores the groups of 16 columns k, k + ns ..; every CTA pushes its part of them, its references and its sums there, over the operands, which nobody
        // needs any more behind the first barrier: [source][group][column][row].  (Pulled by the merging CTA, peer by peer, they took 14 k cycles of a short turn's 48.)
        cg::cluster_group cluster = cg::this_cluster();
        const int groups = (D / 16 + ns - 1) / ns, r = (warp & 3) * 32 + lane;
        float* part = reinterpret_cast<float*>(sm);
        float* stat = part + ns * groups * 2048;                     // [source][reference, sum][row]
        cluster.sync();
        if (warp >= 4) {
            if (n_walk > 0) {
#pragma unroll 1
                for (int c = 0, to = 0, g = 0; c < D; c += 16) {
                    uint32_t w[16];
                    tmem_ld16_async(tmem + ((uint32_t)((warp & 3) * 32) << 16) + c, w);
                    float* dst = cluster.map_shared_rank(part, to) + (rank * groups + g) * 2048 + r;
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) dst[j * 128] = __uint_as_float(w[j]);
                    if (++to == ns) { to = 0; ++g; }
                }
            }
#pragma unroll 1
            for (int k = 0; k < ns; ++k) {
                float* dst = cluster.map_shared_rank(stat, k) + rank * 256 + r;
                dst[0] = m_row; dst[128] = l_row;
            }
        }
        cluster.sync();
        if (warp >= 4) {
            float M = -INFINITY, L = 0.f;
#pragma unroll 1
            for (int k = 0; k < ns; ++k) M = fmaxf(M, stat[k * 256 + r]);
            auto factor = [&](int k) { const float m = stat[k * 256 + r]; return m == -INFINITY ? 0.f : exp2f(m - M); };
#pragma unroll 1
            for (int k = 0; k < ns; ++k) L += stat[k * 256 + 128 + r] * factor(k);
            store(rank * 16, 16 * ns, M, L, r, [&](int c, float* v) {
                const float* p = part + (c / 16) / ns * 2048 + r;
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = 0.f;
#pragma unroll 1
                for (int k = 0; k < ns; ++k, p += groups * 2048) {
                    const float f = factor(k);
                    if (f > 0.f) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] = fmaf(p[j * 128], f, v[j]);
                    }
                }
            });
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 2) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

template <int D, bool SPLIT, bool CAUSAL, bool PAGED>
static int ftc_launch_t(cudaStream_t st, const FlashArgs& a) {
    using C = FtcCfg<D, SPLIT>;
    FtcMaps m;
    // (a pool's rows are addressed through its pages, always inside it: the map's row count only has to reach that far)
    const bf16 *k = PAGED ? a.k_pool : a.k, *v = PAGED ? a.v_pool : a.v;
    const uint64_t rows = PAGED ? (uint64_t)1 << 28 : (uint64_t)a.kv_rows, cols = PAGED ? D : (uint64_t)a.nkv * D, ld = PAGED ? D : (uint64_t)a.kv_stride;
    for (int p = 0; p < 2; ++p) {
        const long long off = p && SPLIT ? a.kv_lo_off : 0;
        if (!tc_tmap_16(&m.k[p], k + off, rows, cols, ld, 64, 64, CU_TENSOR_MAP_SWIZZLE_128B)) return -1001;
        if (!tc_tmap_16(&m.v[p], v + off, rows, cols, ld, C::RB, 64, CU_TENSOR_MAP_SWIZZLE_128B)) return -1001;
    }
    static SmemOptIn seen;
    if (const int e = ensure_dyn_smem(flash_tc_kernel<D, SPLIT, CAUSAL, PAGED>, (size_t)C::SMEM, seen)) return e;
    int* err = nullptr;
    if (const int e = tc_err_word(st, &err)) return e;
    const int max_len = a.seq_len ? a.max_len : a.S, qt = (max_len + 127) / 128;
    // too few query tiles for the chip (a short turn behind a long cached prefix): clusters share their keys, at least two tiles each
    int ns = 1;
    if (!a.seq_len) {
        const int ctas = a.nh * qt, tiles = ((CAUSAL ? a.kv_offset : 0) + a.S + C::BN - 1) / C::BN;
        ns = std::max(1, std::min(std::min(8, tc_device_sms() / ctas), tiles / 2));
        while (ns > 1 && tc_max_clusters(ns) < ctas) --ns;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.nh * ns, qt, a.seq_len ? a.nseq : 1); cfg.blockDim = dim3(256); cfg.dynamicSmemBytes = C::SMEM; cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (ns > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = ns; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = 1;
        ++na;
    }
    if (prefill_pdl()) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = attr; cfg.numAttrs = na;
    return (int)cudaLaunchKernelEx(&cfg, flash_tc_kernel<D, SPLIT, CAUSAL, PAGED>, m, a, ns, err);
}

bool flash_tc_fits(int D, bool causal, bool paged, const FlashArgs& a) {
    if (causal != paged || (!paged && a.kv_rows <= 0) || (D != 64 && D != 128 && !(D == 256 && causal))) return false;
    const long long al = (long long)a.q_stride | a.o_stride | (paged ? 0 : a.kv_stride) | a.q_lo_off | a.kv_lo_off | a.out_lo_off;
    const uintptr_t ptr = (uintptr_t)a.q | (uintptr_t)a.out | (uintptr_t)(paged ? a.k_pool : a.k) | (uintptr_t)(paged ? a.v_pool : a.v);
    return (al & 7) == 0 && (ptr & 15) == 0 && (!a.gate || a.gate_heads || (a.g_stride & 1) == 0);
}
int flash_tc_launch(cudaStream_t st, int D, bool causal, const FlashArgs& a) {
    const bool split = a.q_lo_off != 0;
    if (causal) {
        switch (D) {
            case 64:  return split ? ftc_launch_t<64, true, true, true>(st, a) : ftc_launch_t<64, false, true, true>(st, a);
            case 128: return split ? ftc_launch_t<128, true, true, true>(st, a) : ftc_launch_t<128, false, true, true>(st, a);
            case 256: return split ? ftc_launch_t<256, true, true, true>(st, a) : ftc_launch_t<256, false, true, true>(st, a);
        }
    } else {
        switch (D) {
            case 64:  return split ? ftc_launch_t<64, true, false, false>(st, a) : ftc_launch_t<64, false, false, false>(st, a);
            case 128: return split ? ftc_launch_t<128, true, false, false>(st, a) : ftc_launch_t<128, false, false, false>(st, a);
        }
    }
    return -1000;
}

}  // namespace cb
