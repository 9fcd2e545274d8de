// Linears of few activation rows (M <= 128):  C[M, N] (+)= (A_0 + .. + A_{P-1})[M, K] x W[N, K]^T, the activations as P = 1 .. 3 bf16 planes.
//
// What bounds it is the weight bytes, which pass once whatever M is, so the tile is the weights': 128 weight rows are the MMA's M, and the planes of all
// activation rows side by side are its N (P x M rounded up to 16 columns: a batch of 32 in three planes is one MMA of 96 columns); every plane has
// accumulator columns of its own, added when they are read.  Three planes carry all 24 bits of an f32 activation (a decode batch keeps the
// accuracy of the f32 GEMV it replaces), two the split-precision operands of the prefill, one plain bf16.
//
// A stage is 128 weight rows x 64 CH columns and the planes beside it.  CH = 2, eight MMAs per wait and commit, while three such stages fit (a wait costs
// the issuing warp as much as four MMAs of these widths: tc.cuh, elect_one); CH = 1 for wider activations, whose MMAs take longer anyway:
// with two stages in flight instead of five, 12288 x 2048 at 77 rows in two planes took 43 us.  
//
// Fewer tiles than SMs (N < 19 000): a cluster of up to eight CTAs shares a tile along K and adds its partial tiles through distributed shared memory,
// every CTA finishing its share of the columns.  More: stream-K over (tile, step), the same number of steps on every SM; partial tiles
// go through global memory and the last contributor to arrive adds them, in contributor order either way.
#include "gemm.cuh"
#include "tc.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace cb {
namespace cg = cooperative_groups;

constexpr int GR_MAX_CTAS = 160;
constexpr int GR_TILE = 128 * 128;                // one 64-wide tile of the weights
constexpr int GR_BUDGET = 208 * 1024;
constexpr int GR_EPI = 8;                         // epilogue warps: two take turns at a quarter's chunks of 16 rows

struct GemmRowsArgs {
    GemmEpi ep;
    int M, Mp, N, KB, nstg;        // Mp: M rounded up to 16; KB: steps of 64 CH columns
    int cl;                        // CTAs per tile (a cluster; 1: none), 0: stream-K
    TcSched sc;
    int* err;
};

// one chunk of 16 activation rows m0 .. m0 + 15 of this lane's weight row n
template <int MODE>
__device__ __forceinline__ void rows_epi16(const GemmEpi& ep, int M, int N, int m0, int n, float* v, int lane) {
    const bool in = n < N;
    const int rows = min(16, M - m0);
    if (ep.bias && in) {
        const float b = ep.bias[n];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] += b;
    }
    if (ep.col_scale && in) {
        const float c = ep.col_scale[n];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] *= c;
    }
    if (ep.gate && in) {
        const float gb = ep.gate_bias ? ep.gate_bias[n] : 0.f;
        const float* g = ep.gate + (size_t)m0 * ep.ldg + n;
#pragma unroll
        for (int j = 0; j < 16; ++j) if (j < rows) v[j] *= 1.f / (1.f + expf(-(g[(size_t)j * ep.ldg] + gb)));
    }
    if constexpr (MODE == EPI_STORE_F32 || MODE == EPI_RESID_F32) {
        if (!in) return;
        float* o = reinterpret_cast<float*>(ep.out) + (size_t)m0 * ep.ldo + n;
        if constexpr (MODE == EPI_RESID_F32) {
            float x[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) x[j] = j < rows ? o[(size_t)j * ep.ldo] : 0.f;
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] += x[j];
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) if (j < rows) o[(size_t)j * ep.ldo] = v[j];
    } else if constexpr (MODE == EPI_SILU_MUL_F32 || MODE == EPI_SILU_MUL_BF16) {
        // rows interleaved (gate_j, up_j): an even lane has the gates of a column's 16 rows, its neighbour the ups.  They trade halves: the even lane finishes rows
        // 0 - 7, the odd one 8 - 15, eight independent exponentials and divisions each.
        const bool odd = lane & 1;
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = j < rows ? v[j] : 1.f;       // rows behind the last are zeros, which the division takes 100 cycles each for
        float r[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float x = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 8], 1);
            r[j] = odd ? x : v[j];
            v[j] = odd ? v[j + 8] : x;
        }
        if (ep.glu_limit == 0.f) {
#pragma unroll
            for (int j = 0; j < 8; ++j) r[j] = silu_f(r[j]) * v[j];
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) r[j] = glu_pair_f(r[j], v[j], ep.glu_limit);
        }
        const int mo = m0 + (odd ? 8 : 0);
        if constexpr (MODE == EPI_SILU_MUL_F32) {
#pragma unroll
            for (int j = 0; j < 8; ++j) if (in && mo + j < M) reinterpret_cast<float*>(ep.out)[(size_t)(mo + j) * ep.ldo + (n >> 1)] = r[j];
        } else {
            // neighbouring columns (lanes two apart) as 4-byte stores: the lower lane takes the first four of the rows, the upper the last
            const bool up = lane & 2;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float x = __shfl_xor_sync(0xffffffffu, up ? r[j] : r[j + 4], 2);
                const float a = up ? x : r[j], b = up ? r[j + 4] : x;
                const int m = mo + (up ? 4 : 0) + j;
                if (in && m < M) {
                    uint32_t hi, lo;
                    split_bf16x2(a, b, hi, lo);
                    const size_t off = (size_t)m * ep.ldo + ((n >> 1) & ~1);
                    *reinterpret_cast<uint32_t*>(reinterpret_cast<bf16*>(ep.out) + off) = hi;
                    if (ep.out_lo) *reinterpret_cast<uint32_t*>(reinterpret_cast<bf16*>(ep.out_lo) + off) = lo;
                }
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            if constexpr (MODE == EPI_GELU_ERF_BF16) v[j] = gelu_erf_f(v[j]);
            else if constexpr (MODE == EPI_GELU_TANH_BF16) v[j] = gelu_tanh_f(v[j]);
            else if constexpr (MODE == EPI_RELU2_BF16) { v[j] = fmaxf(v[j], 0.f); v[j] *= v[j]; }
        }
        // neighbouring columns as 4-byte stores: the even lane takes rows 0 - 7, the odd one 8 - 15
        const bool odd = lane & 1;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float x = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 8], 1);
            const float a = odd ? x : v[j], b = odd ? v[j + 8] : x;
            const int jj = j + (odd ? 8 : 0);
            if (in && jj < rows) {
                uint32_t hi, lo;
                split_bf16x2(a, b, hi, lo);
                const size_t off = (size_t)(m0 + jj) * ep.ldo + (n & ~1);
                *reinterpret_cast<uint32_t*>(reinterpret_cast<bf16*>(ep.out) + off) = hi;
                if (ep.out_lo) *reinterpret_cast<uint32_t*>(reinterpret_cast<bf16*>(ep.out_lo) + off) = lo;
            }
        }
    }
}

//   warp 0: TMA producer    warp 1: MMA issuer    warp 2: TMEM allocator    warps 4 - 11: epilogue (TMEM lanes 32 (warp % 4) .., every other 16 rows)
template <int P, int MODE, int CH>
__global__ void __launch_bounds__(128 + 32 * GR_EPI, 1)
gemm_rows_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmA1,
                 const __grid_constant__ CUtensorMap tmA2, GemmRowsArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full[8], empty[8], d_full[2], d_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int last_flag, gave_up;
    const TcWait wait{&gave_up, a.err};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int Mp = a.Mp, KB = a.KB, nstg = a.nstg, cols = P * Mp, stg_bytes = CH * (GR_TILE + cols * 128);
    const int rank = a.cl > 1 ? blockIdx.x % a.cl : 0, t0 = a.cl ? blockIdx.x / a.cl * KB : 0;
    const int it_begin = a.cl ? t0 + rank * KB / a.cl : sched_start(a.sc, blockIdx.x), it_end = a.cl ? t0 + (rank + 1) * KB / a.cl : sched_start(a.sc, blockIdx.x + 1);

    if (threadIdx.x == 0) {
        gave_up = 0;
        for (int i = 0; i < nstg; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&d_full[i], 1); mbar_init(&d_empty[i], GR_EPI); }
        fence_barrier_init();
    }
    if (warp == 2) { tmem_alloc(&tmem_slot, 512); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_launch_dependents();

    if (warp == 0) {
        if (lane == 0) {
            tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmA0);
            auto weights = [&](int it, int st) {
                mbar_arrive_expect_tx(&full[st], stg_bytes);
                const int n0 = it / KB * 128, k0 = it % KB * (64 * CH);
#pragma unroll
                for (int c = 0; c < CH; ++c) tma_load_2d(sm + st * stg_bytes + c * GR_TILE, &tmW, &full[st], k0 + 64 * c, n0);
            };
            // weights do not depend on the predecessor kernel: the first stages' go out before the dependency wait
            const int npre = a.ep.w_dynamic ? 0 : min(it_end - it_begin, nstg);
            for (int i = 0; i < npre; ++i) weights(it_begin + i, i);
            pdl_wait();
            int st = 0; uint32_t ph = 0;
            for (int it = it_begin; it < it_end; ++it) {
                if (it - it_begin >= npre) { wait(&empty[st], ph ^ 1); weights(it, st); }
                const int k0 = it % KB * (64 * CH);
                uint8_t* b = sm + st * stg_bytes + CH * GR_TILE;
#pragma unroll
                for (int c = 0; c < CH; ++c) {
                    tma_load_2d(b + c * cols * 128, &tmA0, &full[st], k0 + 64 * c, 0);
                    if (P > 1) tma_load_2d(b + c * cols * 128 + Mp * 128, &tmA1, &full[st], k0 + 64 * c, 0);
                    if (P > 2) tma_load_2d(b + c * cols * 128 + 2 * Mp * 128, &tmA2, &full[st], k0 + 64 * c, 0);
                }
                if (++st == nstg) { st = 0; ph ^= 1; }
            }
            wait.drain();
        }
    } else if (warp == 1) {
        const uint32_t idesc = make_idesc_bf16(128, cols);
        int st = 0, seg = 0; uint32_t ph = 0;
        for (int it = it_begin; it < it_end; ++seg) {
            const int seg_end = min(it_end, (it / KB + 1) * KB), b = seg & 1;
            wait(&d_empty[b], ((seg >> 1) & 1) ^ 1);
            tc_fence_after();
            const uint32_t d = tmem + (uint32_t)(b * 256);
            for (int i = it; i < seg_end; ++i) {
                wait(&full[st], ph);
                tc_fence_after();
                const uint32_t wa = smem_u32(sm + st * stg_bytes);
                const uint64_t wd = make_smem_desc_sw128(wa), ad = make_smem_desc_sw128(wa + CH * GR_TILE);
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < 4 * CH; ++k)
                        umma_bf16(d, wd + (uint64_t)((k >> 2) * (GR_TILE / 16) + 2 * (k & 3)), ad + (uint64_t)((k >> 2) * cols * 8 + 2 * (k & 3)), idesc,
                                  (uint32_t)((i != it) | (k != 0)));
                    umma_commit(&empty[st]);
                    if (i == seg_end - 1) umma_commit(&d_full[b]);
                }
                __syncwarp();
                if (++st == nstg) { st = 0; ph ^= 1; }
            }
            it = seg_end;
        }
    } else if (warp >= 4) {
        pdl_wait();                                 // (reads / overwrites activations of the predecessor too)
        const int q = warp & 3, part = (warp - 4) >> 2, row = q * 32 + lane;
        const size_t tile_f = (size_t)128 * Mp;
        int seg = 0;
        for (int it = it_begin; it < it_end; ++seg) {
            const int seg_end = min(it_end, (it / KB + 1) * KB), t = it / KB, n = t * 128 + row, b = seg & 1;
            const bool sole = it % KB == 0 && seg_end - it == KB;
            const uint32_t d = tmem + (uint32_t)(b * 256) + ((uint32_t)(q * 32) << 16);
            wait(&d_full[b], (seg >> 1) & 1);
            tc_fence_after();
            // a cluster's partial tile stays in shared memory, in place of the operands (every MMA of this CTA has read its own)
            float* mine = a.cl > 1 ? reinterpret_cast<float*>(sm) + row : a.sc.ws + (size_t)(2 * blockIdx.x + (it == it_begin ? 0 : 1)) * tile_f + row;
#pragma unroll 1
            for (int c = 16 * part; c < Mp; c += 4 * GR_EPI) {
                uint32_t r0[16], r1[16], r2[16];
                tmem_ld16_async(d + c, r0);
                if (P > 1) tmem_ld16_async(d + Mp + c, r1);
                if (P > 2) tmem_ld16_async(d + 2 * Mp + c, r2);
                tmem_ld_wait();
                float v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) {      // small terms first
                    v[j] = __uint_as_float(r0[j]);
                    if (P == 2) v[j] += __uint_as_float(r1[j]);
                    if (P == 3) v[j] += __uint_as_float(r1[j]) + __uint_as_float(r2[j]);
                }
                if (sole) rows_epi16<MODE>(a.ep, a.M, a.N, c, n, v, lane);
                else {
#pragma unroll
                    for (int j = 0; j < 16; ++j) mine[(size_t)(c + j) * 128] = v[j];
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&d_empty[b]);
            if (!sole && a.cl == 0) {               // arrive at the tile; the last of its contributors adds them in order and finishes it
                __threadfence();
                named_bar_sync(1, 32 * GR_EPI);
                const int c_first = sched_owner(a.sc, t * KB), c_last = sched_owner(a.sc, t * KB + KB - 1);
                if (threadIdx.x == 128) last_flag = atomicAdd(&a.sc.counters[t], 1) == c_last - c_first;
                named_bar_sync(1, 32 * GR_EPI);
                if (last_flag) {
                    __threadfence();
#pragma unroll 1
                    for (int c = 16 * part; c < Mp; c += 4 * GR_EPI) {
                        float v[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] = 0.f;
                        for (int cc = c_first; cc <= c_last; cc += 2) {           // two contributors' loads in flight; the additions stay in order
                            const float* p0 = a.sc.ws + (size_t)(2 * cc + (sched_start(a.sc, cc) < t * KB ? 1 : 0)) * tile_f + (size_t)c * 128 + row;
                            const bool two = cc < c_last;
                            const float* p1 = two ? a.sc.ws + (size_t)(2 * (cc + 1) + (sched_start(a.sc, cc + 1) < t * KB ? 1 : 0)) * tile_f + (size_t)c * 128 + row : p0;
                            float x0[16], x1[16];
#pragma unroll
                            for (int j = 0; j < 16; ++j) x0[j] = __ldcg(p0 + j * 128);
#pragma unroll
                            for (int j = 0; j < 16; ++j) x1[j] = two ? __ldcg(p1 + j * 128) : 0.f;
#pragma unroll
                            for (int j = 0; j < 16; ++j) v[j] += x0[j];
                            if (two) {
#pragma unroll
                                for (int j = 0; j < 16; ++j) v[j] += x1[j];
                            }
                        }
                        rows_epi16<MODE>(a.ep, a.M, a.N, c, n, v, lane);
                    }
                    if (threadIdx.x == 128) a.sc.counters[t] = 0;
                }
                named_bar_sync(1, 32 * GR_EPI);             // last_flag is rewritten by the next segment
            }
            it = seg_end;
        }
    }
    if (a.cl > 1) {
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        if (warp >= 4) {
            const int row = (warp & 3) * 32 + lane, n = it_begin / KB * 128 + row;
#pragma unroll 1
            for (int c = (rank + ((warp - 4) >> 2) * a.cl) * 16; c < Mp; c += 4 * GR_EPI * a.cl) {
                float v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = 0.f;
                for (int r = 0; r < a.cl; ++r) {
                    const float* p = cluster.map_shared_rank(reinterpret_cast<float*>(sm), r) + (size_t)c * 128 + row;
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] += p[j * 128];
                }
                rows_epi16<MODE>(a.ep, a.M, a.N, c, n, v, lane);
            }
        }
        cluster.sync();                              // nobody leaves while its shared memory is still being read
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 2) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// CTAs per tile: as many as the chip has room for at once (clusters live inside a GPC: sixteen of eight CTAs do not fit, and a second wave
// doubled 2048 x 6144 at 77 rows to 37 us), each with at least 256 columns of K (`steps` of 64)
static int rows_cluster(int tiles_n, int steps, int sms) {
    int cl = std::max(1, std::min(std::min(8, sms / tiles_n), steps / 4));
    while (cl > 1 && tc_max_clusters(cl) < tiles_n) --cl;
    return cl;
}

// Is this kernel the faster one of the two for up to 128 rows?  Both stream the weights at about the same rate; the tiles of gemm.cu pay for 128 rows whatever M
// is, while here the activations' traffic and the epilogue grow with the rows.  us, here / gemm.cu (planes x rows: weights):
//   f32, a cluster per tile    always, but for 1 x 96 - 128 of K = 1024: 4096 x 1024 8.3 / 8.0 (1 x 77: 8.0 / 7.9; 4096 x 2048 11.3 / 12.0; 2 x 128: 4096 x 1024 10.0 / 10.2)
//   f32, one CTA per tile      1 x 80: 12288 x 2048 10.9 / 12.9, 24576 x 4096 41.3 / 41.4; 1 x 96: 11.2 / 12.9, 43.3 / 41.8; 2 x 64: 16.7 / 17.7, 44.2 / 53.9; 2 x 96: 16384 x 2048
//                              17.7 / 17.8, 24576 x 4096 47.1 / 54.1; 2 x 128: 18.3 / 18.1, 52.3 / 54.5
//   gate / up, one plane       a cluster: 64 rows 6144 x 1024 7.9 / 9.0, 7168 x 1024 8.4 / 9.4; 77: 9.3 / 9.0, 10.0 / 10.1.  One CTA: 77 12288 x 2048 14.7 / 16.1, 24576 x 4096
//                              43.2 / 44.4; 96: 15.4 / 16.2, 45.5 / 45.0
//   gate / up, two planes      96 rows: 6144 x 1024 11.0 / 11.1, 12288 x 2048 19.9 / 20.6; 112: 11.6 / 11.2, 21.2 / 20.7; more tiles than SMs: 128 24576 x 4096 63.2 / 63.9
//   other bf16 results         a cluster: 1 x 96 4096 x 1024 9.3 / 9.5, 112 10.2 / 9.6, 128 4096 x 2048 11.9 / 12.2; 2 x 128: 4096 x 1024 11.8 / 12.5
//                              one CTA: 1 x 48: 12288 x 2048 10.9 / 12.8, 24576 x 4096 38.8 / 40.5; 1 x 64: 11.1 / 12.8, 39.6 / 40.9; 1 x 80: 11.7 / 12.9, 41.7 / 40.9; 2 x 48:
//                              12.1 / 17.6, 40.4 / 51.9; 2 x 64: 17.3 / 17.8, 45.0 / 52.0; 2 x 80: 18.2 / 17.9, 46.9 / 52.1
// (One CTA per tile: measured back to back after either kernel got eight epilogue warps and the tiles lost their divisions.  The lines are those from before and lie on
// the safe side: two f32 planes could go to 96 rows, other bf16 results to 64.)
bool gemm_rows_pays(int mode, int P, int M, int N, int K) {
    if (M > 128) return false;
    const bool f32 = mode == EPI_STORE_F32 || mode == EPI_RESID_F32, glu = mode == EPI_SILU_MUL_BF16;
    const int tiles_n = (N + 127) / 128, sms = std::min(tc_device_sms(), GR_MAX_CTAS), cl = tiles_n <= sms ? rows_cluster(tiles_n, K / 64, sms) : 1;
    if (glu) return M <= (P == 1 ? (cl > 1 ? 64 : 80) : tiles_n <= sms ? 96 : 128);
    if (cl == 1) return M <= (!f32 ? 48 : P == 1 ? 80 : 64);
    return P > 1 || K > 1024 || M <= (f32 ? 80 : 96);
}

template <int P, int MODE, int CH>
static int rows_launch_c(cudaStream_t st, const bf16* const* A, int lda, const bf16* W, int M, int N, int K, const GemmEpi& ep, bool pdl) {
    GemmRowsArgs a = {};
    a.ep = ep; a.M = M; a.Mp = (M + 15) / 16 * 16; a.N = N; a.KB = (K + 64 * CH - 1) / (64 * CH);
    CUtensorMap tmW, tm[3];
    if (!tc_tmap_bf16(&tmW, W, (uint64_t)N, (uint64_t)K, (uint64_t)K, 128)) return -1001;
    for (int p = 0; p < 3; ++p)
        if (!tc_tmap_bf16(&tm[p], A[p < P ? p : 0], (uint64_t)M, (uint64_t)K, (uint64_t)lda, (uint32_t)a.Mp)) return -1001;
    const int stg = CH * (GR_TILE + P * a.Mp * 128);
    a.nstg = std::min(8, GR_BUDGET / stg);
    static SmemOptIn seen;
    const size_t smem = (size_t)a.nstg * stg + 1024;
    if (const int e = ensure_dyn_smem(gemm_rows_kernel<P, MODE, CH>, smem, seen)) return e;
    TcSched& sc = a.sc;
    sc.tiles_m = 1; sc.tiles_n = (N + 127) / 128; sc.KB = a.KB;
    const long long iters = (long long)sc.tiles_n * a.KB;
    if (iters > 0x7fffffffLL) return -1000;
    const int sms = std::min(tc_device_sms(), GR_MAX_CTAS);
    int grid;
    if (sc.tiles_n <= sms) {
        a.cl = rows_cluster(sc.tiles_n, a.KB * CH, sms);
        grid = sc.tiles_n * a.cl;
        if (const int e = tc_err_word(st, &a.err)) return e;
    } else {
        TcScratch s;
        if (const int e = tc_scratch_get(st, sc.tiles_n, &s)) return e;
        sc.ws = s.ws; sc.counters = s.counters; a.err = s.err;
        sc.unit = 1; sc.G = sms;
        sc.base = (int)(iters / sc.G); sc.rem = (int)(iters % sc.G);
        grid = sc.G;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid); cfg.blockDim = dim3(128 + 32 * GR_EPI); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (a.cl > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = a.cl; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = 1;
        ++na;
    }
    if (pdl) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = attr; cfg.numAttrs = na;
    return (int)cudaLaunchKernelEx(&cfg, gemm_rows_kernel<P, MODE, CH>, tmW, tm[0], tm[1], tm[2], a);
}

template <int P, int MODE>
static int rows_launch_t(cudaStream_t st, const bf16* const* A, int lda, const bf16* W, int M, int N, int K, const GemmEpi& ep, bool pdl) {
    return P * ((M + 15) / 16 * 16) <= 96 ? rows_launch_c<P, MODE, 2>(st, A, lda, W, M, N, K, ep, pdl) : rows_launch_c<P, MODE, 1>(st, A, lda, W, M, N, K, ep, pdl);
}

template <int MODE>
static int rows_launch_m(cudaStream_t st, const bf16* const* A, int P, int lda, const bf16* W, int M, int N, int K, const GemmEpi& ep, bool pdl) {
    switch (P) {
        case 1: return rows_launch_t<1, MODE>(st, A, lda, W, M, N, K, ep, pdl);
        case 2: return rows_launch_t<2, MODE>(st, A, lda, W, M, N, K, ep, pdl);
        default: return -1000;
    }
}

int gemm_rows_launch(cudaStream_t st, const bf16* const* A, int P, int lda, const bf16* W, int M, int N, int K, const GemmEpi& ep, bool pdl) {
    // f32 results leave one by one, bf16 ones in pairs of columns; of SiLU's (gate, up) rows a result takes two
    const int unit = ep.mode == EPI_STORE_F32 || ep.mode == EPI_RESID_F32 ? 1 : ep.mode == EPI_SILU_MUL_BF16 ? 4 : 2;
    if (M < 1 || P * ((M + 15) / 16 * 16) > 256 || N <= 0 || K <= 0 || (K % 8) != 0 || (N % unit) != 0 || (lda % 8) != 0) return -1000;
    if (P == 3) {                                   // the decode batch's epilogues
        switch (ep.mode) {
            case EPI_STORE_F32:    return rows_launch_t<3, EPI_STORE_F32>(st, A, lda, W, M, N, K, ep, pdl);
            case EPI_RESID_F32:    return rows_launch_t<3, EPI_RESID_F32>(st, A, lda, W, M, N, K, ep, pdl);
            case EPI_SILU_MUL_F32: return rows_launch_t<3, EPI_SILU_MUL_F32>(st, A, lda, W, M, N, K, ep, pdl);
            default: return -1000;
        }
    }
    switch (ep.mode) {
        case EPI_STORE_F32:      return rows_launch_m<EPI_STORE_F32>(st, A, P, lda, W, M, N, K, ep, pdl);
        case EPI_STORE_BF16:     return rows_launch_m<EPI_STORE_BF16>(st, A, P, lda, W, M, N, K, ep, pdl);
        case EPI_RESID_F32:      return rows_launch_m<EPI_RESID_F32>(st, A, P, lda, W, M, N, K, ep, pdl);
        case EPI_SILU_MUL_BF16:  return rows_launch_m<EPI_SILU_MUL_BF16>(st, A, P, lda, W, M, N, K, ep, pdl);
        case EPI_GELU_ERF_BF16:  return rows_launch_m<EPI_GELU_ERF_BF16>(st, A, P, lda, W, M, N, K, ep, pdl);
        case EPI_GELU_TANH_BF16: return rows_launch_m<EPI_GELU_TANH_BF16>(st, A, P, lda, W, M, N, K, ep, pdl);
        case EPI_RELU2_BF16:     return rows_launch_m<EPI_RELU2_BF16>(st, A, P, lda, W, M, N, K, ep, pdl);
        default: return -1000;
    }
}

// f32 rows -> three bf16 planes (hi, mid, lo: all 24 bits), RMS-normalised first when norm_w is set.  One CTA per row; a few microseconds of latency.
__global__ void __launch_bounds__(256)
rows_split3_kernel(const float* __restrict__ x, int ldx, int K, const float* __restrict__ norm_w, float eps, bf16* __restrict__ out, long long plane) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ float red[32];
    const float* xr = x + (size_t)blockIdx.x * ldx;
    float rstd = 1.f;
    if (norm_w) {
        float ssq = 0.f;
        for (int i = threadIdx.x * 4; i < K; i += 1024) {
            const float4 v = *reinterpret_cast<const float4*>(xr + i);
            ssq += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
        }
        rstd = rsqrtf(block_sum(ssq, red) / (float)K + eps);
    }
    bf16* o = out + (size_t)blockIdx.x * K;
    for (int i = threadIdx.x * 4; i < K; i += 1024) {
        float4 v = *reinterpret_cast<const float4*>(xr + i);
        if (norm_w) {
            const float4 g = *reinterpret_cast<const float4*>(norm_w + i);
            v.x = v.x * rstd * g.x; v.y = v.y * rstd * g.y; v.z = v.z * rstd * g.z; v.w = v.w * rstd * g.w;
        }
        uint32_t h[2], m[2], l[2];
        const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const float a = e[2 * k], b = e[2 * k + 1];
            h[k] = pack_bf16(a, b);
            const float ra = a - bf16lo(h[k]), rb = b - bf16hi(h[k]);
            m[k] = pack_bf16(ra, rb);
            l[k] = pack_bf16(ra - bf16lo(m[k]), rb - bf16hi(m[k]));
        }
        *reinterpret_cast<uint2*>(o + i) = make_uint2(h[0], h[1]);
        *reinterpret_cast<uint2*>(o + plane + i) = make_uint2(m[0], m[1]);
        *reinterpret_cast<uint2*>(o + 2 * plane + i) = make_uint2(l[0], l[1]);
    }
}
int rows_split3_launch(cudaStream_t st, const float* x, int ldx, int M, int K, const float* norm_w, float eps, bf16* out, long long plane, bool pdl) {
    if ((K % 4) != 0 || (ldx % 4) != 0 || M < 1) return -1000;
    return launch_k(rows_split3_kernel, dim3(M), dim3(256), 0, st, pdl, x, ldx, K, norm_w, eps, out, plane);
}

}  // namespace cb
