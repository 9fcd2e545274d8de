// Decode-path kernels.  See decode.cuh for the design.
#include "decode.cuh"
#include "tc.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace cb {

// =====================================================================================
// Weight-streaming GEMV:  y[b, n] = epilogue( sum_k W[n, k] * x[b, k] )          (B <= 4 sequences)
//
// grid = #SMs; CTA c owns the contiguous rows [c*rpc, (c+1)*rpc) of W.  A unit of work is four rows x one of `ns` slices of K (gemv_slices): a warp takes
// every GV_WARPS-th unit and runs its own, barrier-free pipeline: slots of 4 rows x 256 columns (2 KB) filled by cp.async (16 B per lane, L1-bypassing),
// every lane reading back what it copied itself, into f32 FMAs.  Four rows share each read of the activations (f32 in shared memory, RMSNorm folded in):
// row by row they were two thirds of the shared-memory traffic, which bound the kernel wherever the weights had come early.  A unit's sums are reduced
// over the warp together (6 shuffles for four rows of one sequence instead of 20) and a row's slices added in order, so results repeat bit for bit.
// Weights do not depend on the previous kernel, so the pipelines are primed BEFORE griddepcontrol.wait, and the HBM pipe stays busy across the boundary.
// What is left per launch: 0.7 us from one grid's end to the next one's wait, 0.7 for the activations' round trip to the L2 (a chain of kernels
// that only do that takes 1.4 us each).  In a chain of its own kind, us, before / after: 4096 x 1024 4.0 / 3.5, 6144 x 1024 (gate / up) 5.4 / 4.3,
// 12288 x 2048 10.6 / 9.3, 24576 x 4096 31.7 / 30.3.  (Two CTAs per SM, so that the next launch's sit there early, gained nothing and cost the long ones 10 %.)
// Epilogue (all threads): store / residual add / SiLU*up on interleaved rows / logits + CTA argmax.
// =====================================================================================
constexpr int GV_WARPS = 16;
constexpr int GV_ROWS = 4;                             // rows of a unit
constexpr int GV_SLOT = GV_ROWS * 512;
constexpr int GV_THREADS = GV_WARPS * 32;
__host__ __device__ constexpr int gv_depth(int B) { return B == 1 ? 4 : 2; }          // batched activations take the ring's shared memory

__device__ __forceinline__ void cp_async16_cg(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit_g() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait_g() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// The streams' form of the staged input: a thread takes four columns of every stream at a time.  Returns its share of the sum of squares.
template <int S>
__device__ __forceinline__ float gemv_stage_streams(const GemvArgs& a, int b, float4* xs, int K8, bool keep) {
    const float* x = a.fs_x + (size_t)b * S * a.K;
    const float* y = a.fs_y + (size_t)b * a.K;
    float* nx = a.fs_next + (size_t)b * S * a.K;
    float ssq = 0.f;
    for (int q = threadIdx.x; q < 2 * K8; q += GV_THREADS) {
        const float4 yv = reinterpret_cast<const float4*>(y)[q], w = reinterpret_cast<const float4*>(a.norm_w)[q];
        float4 xv[S], u = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int s = 0; s < S; ++s) xv[s] = reinterpret_cast<const float4*>(x + (size_t)s * a.K)[q];
#pragma unroll
        for (int t = 0; t < S; ++t) {
            const float o = a.fs_w[t], c = a.fs_in[t];
            float4 n = make_float4(o * yv.x, o * yv.y, o * yv.z, o * yv.w);
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const float m = a.fs_mix[s * S + t];
                n.x = fmaf(m, xv[s].x, n.x); n.y = fmaf(m, xv[s].y, n.y); n.z = fmaf(m, xv[s].z, n.z); n.w = fmaf(m, xv[s].w, n.w);
            }
            u.x = fmaf(c, n.x, u.x); u.y = fmaf(c, n.y, u.y); u.z = fmaf(c, n.z, u.z); u.w = fmaf(c, n.w, u.w);
            if (keep) reinterpret_cast<float4*>(nx + (size_t)t * a.K)[q] = n;
        }
        ssq = fmaf(u.x, u.x, ssq); ssq = fmaf(u.y, u.y, ssq); ssq = fmaf(u.z, u.z, ssq); ssq = fmaf(u.w, u.w, ssq);
        xs[(size_t)(b * 2 + (q & 1)) * K8 + (q >> 1)] = make_float4(u.x * w.x, u.y * w.y, u.z * w.z, u.w * w.w);
    }
    return ssq;
}

// NORM: 0 the input as it is, 1 RMS norm folded in, 2 the norm of a sum of parallel streams
template <int B, int EPI, int NORM>
__global__ void __launch_bounds__(GV_THREADS, 1)
gemv_kernel(GemvArgs a, int ns) {
    extern __shared__ __align__(1024) unsigned char gsm[];
    // layout: [rings: GV_WARPS * depth * 2 KB][xs: B * K f32][sums: B * rpc * ns f32]
    const int K8 = a.K >> 3;
    constexpr int ROWS_PER_UNIT = (EPI == GEMV_SILU_MUL) ? 2 : 1;
    const int units = a.N / ROWS_PER_UNIT;
    const int upc = (units + gridDim.x - 1) / gridDim.x;
    const int rpc = upc * ROWS_PER_UNIT;                               // rows per CTA (capacity)
    const int r0 = blockIdx.x * rpc;
    const int r1 = min(a.N, r0 + rpc);
    const int nrows = max(0, r1 - r0);
    constexpr int DEPTH = gv_depth(B);
    float4* xs = reinterpret_cast<float4*>(gsm + GV_WARPS * DEPTH * GV_SLOT);
    float* acc_s = reinterpret_cast<float*>(xs) + (size_t)B * a.K;
    __shared__ float red[B][GV_WARPS];
    __shared__ float rstd_s[B];
    __shared__ float wbest_v[GV_WARPS][B];
    __shared__ int wbest_i[GV_WARPS][B];
    __shared__ int is_last_s;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int chunks = a.K >> 8, work = (nrows + GV_ROWS - 1) / GV_ROWS * ns;           // (K % 256 == 0)
    // a walk over this warp's slots: unit u, column chunk c of [c0, c1)
    struct Walk { int u, row, slice, c, c1; };
    auto start = [&](Walk& w, int u) {
        w.u = u;
        if (u < work) { const int blk = u / ns; w.row = blk * GV_ROWS; w.slice = u - blk * ns; w.c = w.slice * chunks / ns; w.c1 = (w.slice + 1) * chunks / ns; }
    };
    const unsigned char* wbase = reinterpret_cast<const unsigned char*>(a.W) + (size_t)r0 * a.K * 2 + lane * 16;
    unsigned char* ring = gsm + (size_t)warp * DEPTH * GV_SLOT + lane * 16;
    const uint32_t ring_u32 = smem_u32(ring);
    const size_t row_bytes = (size_t)a.K * 2;
    Walk wi;
    start(wi, warp);
    uint32_t islot = 0;
    auto issue = [&]() {
        if (wi.u < work) {
            const unsigned char* src = wbase + (size_t)wi.row * row_bytes + wi.c * 512;
#pragma unroll
            for (int i = 0; i < GV_ROWS; ++i)
                if (wi.row + i < nrows) cp_async16_cg(ring_u32 + islot * GV_SLOT + i * 512, src + i * row_bytes);
            if (++wi.c == wi.c1) start(wi, wi.u + GV_WARPS);
        }
        islot = islot + 1 == DEPTH ? 0 : islot + 1;
        cp_async_commit_g();
    };
    // prime the pipeline: weights do not depend on the previous kernel
#pragma unroll
    for (int g = 0; g < DEPTH; ++g) issue();
    // RMSNorm weights are immutable (and cold in every cache): fetch this thread's first chunk before the dependency wait
    float4 nw0 = make_float4(0.f, 0.f, 0.f, 0.f), nw1 = nw0;
    if (NORM == 1 && tid < K8) { nw0 = reinterpret_cast<const float4*>(a.norm_w)[2 * tid]; nw1 = reinterpret_cast<const float4*>(a.norm_w)[2 * tid + 1]; }

    pdl_wait();
    pdl_launch_dependents();

    // the residual's old values travel beside the activations: read in the epilogue they put another round trip to the L2 (0.5 us) behind the dot products
    float old[B];
    if constexpr (EPI == GEMV_RESID) {
#pragma unroll
        for (int b = 0; b < B; ++b) old[b] = tid < nrows ? a.y[(size_t)b * a.ldy + r0 + tid] : 0.f;
    }
    // --- stage activations (f32) and, if NORM, fold the RMSNorm weight in and get 1/rms ---
#pragma unroll
    for (int b = 0; b < B; ++b) {
        float ssq = 0.f;
        if constexpr (NORM == 2) {                    // (block 0 leaves the new streams)
            const bool keep = blockIdx.x == 0;
            ssq = a.fs_n == 1 ? gemv_stage_streams<1>(a, b, xs, K8, keep) : a.fs_n == 2 ? gemv_stage_streams<2>(a, b, xs, K8, keep) :
                  a.fs_n == 3 ? gemv_stage_streams<3>(a, b, xs, K8, keep) : gemv_stage_streams<4>(a, b, xs, K8, keep);
        } else
        for (int i = tid; i < K8; i += GV_THREADS) {
            const float4* xp = reinterpret_cast<const float4*>(a.x + (size_t)b * a.ldx) + 2 * i;
            float4 lo = xp[0], hi = xp[1];
            if (NORM) {
                ssq += lo.x * lo.x + lo.y * lo.y + lo.z * lo.z + lo.w * lo.w + hi.x * hi.x + hi.y * hi.y + hi.z * hi.z + hi.w * hi.w;
                const float4 w0 = (i == tid) ? nw0 : reinterpret_cast<const float4*>(a.norm_w)[2 * i];
                const float4 w1 = (i == tid) ? nw1 : reinterpret_cast<const float4*>(a.norm_w)[2 * i + 1];
                lo.x *= w0.x; lo.y *= w0.y; lo.z *= w0.z; lo.w *= w0.w;
                hi.x *= w1.x; hi.y *= w1.y; hi.z *= w1.z; hi.w *= w1.w;
            }
            if (!NORM && a.dyt_w != nullptr) {
                const float al = *a.dyt_alpha;
                const float4 w0 = reinterpret_cast<const float4*>(a.dyt_w)[2 * i], w1 = reinterpret_cast<const float4*>(a.dyt_w)[2 * i + 1];
                const float4 b0 = reinterpret_cast<const float4*>(a.dyt_b)[2 * i], b1 = reinterpret_cast<const float4*>(a.dyt_b)[2 * i + 1];
                lo.x = fmaf(tanhf(al * lo.x), w0.x, b0.x); lo.y = fmaf(tanhf(al * lo.y), w0.y, b0.y);
                lo.z = fmaf(tanhf(al * lo.z), w0.z, b0.z); lo.w = fmaf(tanhf(al * lo.w), w0.w, b0.w);
                hi.x = fmaf(tanhf(al * hi.x), w1.x, b1.x); hi.y = fmaf(tanhf(al * hi.y), w1.y, b1.y);
                hi.z = fmaf(tanhf(al * hi.z), w1.z, b1.z); hi.w = fmaf(tanhf(al * hi.w), w1.w, b1.w);
            }
            xs[(size_t)(b * 2 + 0) * K8 + i] = lo;
            xs[(size_t)(b * 2 + 1) * K8 + i] = hi;
        }
        if (NORM) {
            ssq = warp_sum(ssq);
            if (lane == 0) red[b][warp] = ssq;
        }
    }
    __syncthreads();
    // 1 / rms is first read behind the next barrier: a warp per sequence adds the warps' shares while the others start on their rows
    if (NORM && warp < B) {
        const float ms = warp_sum(lane < GV_WARPS ? red[warp][lane] : 0.f) / (float)(a.norm_dim > 0 ? a.norm_dim : a.K) + a.eps;
        if (lane == 0) rstd_s[warp] = NORM == 2 ? 1.f / sqrtf(ms) : rsqrtf(ms);
    }
    if (NORM && a.norm_out != nullptr) __syncthreads();
    if (NORM && a.norm_out != nullptr && blockIdx.x == 0) {      // post-norm hidden state for callers that need it (TTS code predictor input)
#pragma unroll
        for (int b = 0; b < B; ++b)
            for (int i = tid; i < K8; i += GV_THREADS) {
                const float r = rstd_s[b];
                const float4 lo = xs[(size_t)(b * 2 + 0) * K8 + i], hi = xs[(size_t)(b * 2 + 1) * K8 + i];
                float4* o = reinterpret_cast<float4*>(a.norm_out + (size_t)b * a.K) + 2 * i;
                o[0] = make_float4(lo.x * r, lo.y * r, lo.z * r, lo.w * r);
                o[1] = make_float4(hi.x * r, hi.y * r, hi.z * r, hi.w * r);
            }
    }

    {
        constexpr int V = GV_ROWS * B;                      // sums of a unit: value i * B + b is row i of sequence b
        Walk w;
        uint32_t slot = 0;
        for (start(w, warp); w.u < work; start(w, w.u + GV_WARPS)) {
            float acc[V], acc2[V];
#pragma unroll
            for (int v = 0; v < V; ++v) { acc[v] = 0.f; acc2[v] = 0.f; }
            for (; w.c < w.c1; ++w.c) {
                cp_async_wait_g<DEPTH - 1>();               // this slot has landed (groups complete in order); a lane reads its own copies
                uint4 q[GV_ROWS];
#pragma unroll
                for (int i = 0; i < GV_ROWS; ++i) q[i] = *reinterpret_cast<const uint4*>(ring + slot * GV_SLOT + i * 512);
                const int idx = (w.c << 5) + lane;          // 8-element piece of the row
#pragma unroll
                for (int b = 0; b < B; ++b) {
                    const float4 xl = xs[(size_t)(b * 2 + 0) * K8 + idx];
                    const float4 xh = xs[(size_t)(b * 2 + 1) * K8 + idx];
#pragma unroll
                    for (int i = 0; i < GV_ROWS; ++i) {
                        float t = acc[i * B + b], u = acc2[i * B + b];
                        t = fmaf(bf16lo(q[i].x), xl.x, t); u = fmaf(bf16lo(q[i].z), xh.x, u);
                        t = fmaf(bf16hi(q[i].x), xl.y, t); u = fmaf(bf16hi(q[i].z), xh.y, u);
                        t = fmaf(bf16lo(q[i].y), xl.z, t); u = fmaf(bf16lo(q[i].w), xh.z, u);
                        t = fmaf(bf16hi(q[i].y), xl.w, t); u = fmaf(bf16hi(q[i].w), xh.w, u);
                        acc[i * B + b] = t; acc2[i * B + b] = u;
                    }
                }
                issue();                                    // refill the slot just drained
                slot = slot + 1 == DEPTH ? 0 : slot + 1;
            }
            // all V sums over the warp at once: each step halves the values a lane carries on
#pragma unroll
            for (int v = 0; v < V; ++v) acc[v] += acc2[v];
            int id = 0, bit = 16;
#pragma unroll
            for (int n = V / 2; n >= 1; n >>= 1, bit >>= 1) {
                const bool up = lane & bit;
#pragma unroll
                for (int v = 0; v < n; ++v) {
                    const float give = up ? acc[v] : acc[v + n], keep = up ? acc[v + n] : acc[v];
                    acc[v] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
                }
                id += up ? n : 0;
            }
            for (int m = bit; m > 0; m >>= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], m);
            const int row = w.row + id / B, b = id % B;
            if ((lane & (2 * bit - 1)) == 0 && row < nrows) acc_s[((size_t)b * rpc + row) * ns + w.slice] = acc[0];
        }
    }
    __syncthreads();
    auto sum_of = [&](int b, int i) {                       // a row's slices, in order
        const float* p = acc_s + ((size_t)b * rpc + i) * ns;
        float v = p[0];
        for (int k = 1; k < ns; ++k) v += p[k];
        return v;
    };

    // ------------------------------- epilogue (all threads) -------------------------------
    float bestv[B];
    int besti[B];
#pragma unroll
    for (int b = 0; b < B; ++b) { bestv[b] = -INFINITY; besti[b] = 0x7fffffff; }
    if constexpr (EPI == GEMV_SILU_MUL) {
        for (int u = tid; u < nrows / 2; u += GV_THREADS) {
#pragma unroll
            for (int b = 0; b < B; ++b) {
                const float r = NORM ? rstd_s[b] : 1.f;
                float g = sum_of(b, 2 * u) * r, up = sum_of(b, 2 * u + 1) * r;
                if (a.bias) { g += a.bias[r0 + 2 * u]; up += a.bias[r0 + 2 * u + 1]; }
                a.y[(size_t)b * a.ldy + (r0 / 2 + u)] = glu_pair_f(g, up, a.glu_limit);
            }
        }
    } else {
        for (int i = tid; i < nrows; i += GV_THREADS) {
#pragma unroll
            for (int b = 0; b < B; ++b) {
                const float v = sum_of(b, i) * (NORM ? rstd_s[b] : 1.f);
                float* yp = a.y + (size_t)b * a.ldy + r0 + i;
                if constexpr (EPI == GEMV_RESID) {
                    float add = a.bias ? v + a.bias[r0 + i] : v;
                    if (a.out_scale) add *= a.out_scale[r0 + i];
                    if (a.gate) add *= 1.f / (1.f + expf(-(a.gate[(size_t)b * a.ldg + r0 + i] + (a.gate_bias ? a.gate_bias[r0 + i] : 0.f))));
                    *yp = (i == tid ? old[b] : *yp) + add;
                } else if constexpr (EPI == GEMV_RELU2) { const float p = fmaxf(v, 0.f); *yp = p * p; }
                else *yp = v;
                if constexpr (EPI == GEMV_LOGITS_ARGMAX) {
                    if (v > bestv[b]) { bestv[b] = v; besti[b] = r0 + i; }   // a thread's rows ascend: first maximum wins
                }
            }
        }
    }

    if constexpr (EPI == GEMV_LOGITS_ARGMAX) {
        // CTA-level (value, lowest index) reduction, then last-CTA-done finalisation.
#pragma unroll
        for (int b = 0; b < B; ++b) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, bestv[b], o);
                const int oi = __shfl_xor_sync(0xffffffffu, besti[b], o);
                if (ov > bestv[b] || (ov == bestv[b] && oi < besti[b])) { bestv[b] = ov; besti[b] = oi; }
            }
        }
        if (lane == 0) {
#pragma unroll
            for (int b = 0; b < B; ++b) { wbest_v[warp][b] = bestv[b]; wbest_i[warp][b] = besti[b]; }
        }
        __syncthreads();
        if (tid < B) {
            float bv = -INFINITY; int bi = 0x7fffffff;
            for (int w = 0; w < GV_WARPS; ++w) {
                const float v = wbest_v[w][tid]; const int i = wbest_i[w][tid];
                if (v > bv || (v == bv && i < bi)) { bv = v; bi = i; }
            }
            a.part_val[tid * gridDim.x + blockIdx.x] = bv;
            a.part_idx[tid * gridDim.x + blockIdx.x] = bi;
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) {
            const unsigned int t = atomicAdd(a.ticket, 1u);
            is_last_s = (t == gridDim.x - 1);
        }
        __syncthreads();
        if (is_last_s) {
            __threadfence();
            __shared__ uint32_t tok_s[B];
            if (warp < B) {
                const int b = warp;
                float bv = -INFINITY; int bi = 0x7fffffff;
                for (int c = lane; c < (int)gridDim.x; c += 32) {
                    const float v = __ldcg(a.part_val + b * gridDim.x + c);
                    const int i = __ldcg(a.part_idx + b * gridDim.x + c);
                    if (v > bv || (v == bv && i < bi)) { bv = v; bi = i; }
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
                    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                    if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
                }
                if ((unsigned)bi >= (unsigned)a.N) bi = 0;       // an all-NaN row has no maximum: never gather from an out-of-range id
                if (lane == 0) {
                    SeqState* s = a.state + b;
                    if (a.out_tokens) a.out_tokens[(size_t)b * a.out_stride + s->step] = (uint32_t)bi;
                    uint32_t fed = (uint32_t)bi;
                    if (a.force_tokens) fed = a.force_tokens[s->step];
                    if (a.advance == 2) fed = s->token;
                    tok_s[b] = fed;
                    if (a.advance) {
                        s->token = fed;
                        s->kv_len += 1;
                        s->pos[0] += 1; s->pos[1] += 1; s->pos[2] += 1;
                    }
                    s->step += 1;
                }
            }
            if (tid == 0) *a.ticket = 0u;
            __syncthreads();
            if (a.advance && a.embed != nullptr) {   // gather the next step's input embedding (bf16 -> f32 residual stream)
                for (int b = 0; b < B; ++b) {
                    const bf16* row = a.embed + (size_t)tok_s[b] * a.H;
                    for (int i = tid; i < a.H; i += GV_THREADS) a.x_next[(size_t)b * a.H + i] = __bfloat162float(row[i]);
                }
            }
        }
    }
}

static int gemv_rpc(int N, int rows_per_unit, int grid) { return (N / rows_per_unit + grid - 1) / grid * rows_per_unit; }
static size_t gemv_smem_bytes(int B, int K, int rpc, int ns) { return (size_t)GV_WARPS * gv_depth(B) * GV_SLOT + (size_t)B * K * 4 + (size_t)B * rpc * ns * 4 + 16; }
// Shared memory that a launch may ask for: 227 KB a block has, less the norm's own arrays where there is one (with the alignment of what follows them, 1 KB).
constexpr size_t gemv_most(bool norm) { return (norm ? 226 : 227) * 1024; }
// Slices of K a CTA's rows are cut into: the fewest column chunks on the busiest warp (a unit's reduction and its first slot cost about another), while
// the sums fit.  One slice wherever the rows are enough for the warps.
static int gemv_slices(int B, int K, int rpc, bool norm) {
    const int chunks = K / 256, blocks = (rpc + GV_ROWS - 1) / GV_ROWS;
    int best = 1, cost = 1 << 30;
    for (int ns = 1; ns <= std::min(chunks, GV_WARPS); ++ns) {
        if (ns > 1 && gemv_smem_bytes(B, K, rpc, ns) > gemv_most(norm)) break;
        const int c = (blocks * ns + GV_WARPS - 1) / GV_WARPS * ((chunks + ns - 1) / ns + 1);
        if (c < cost) { cost = c; best = ns; }
    }
    return best;
}

template <int B, int EPI, int NORM>
static int gemv_launch_t(cudaStream_t st, const GemvArgs& a, int num_sms, bool pdl) {
    const int rpc = gemv_rpc(a.N, EPI == GEMV_SILU_MUL ? 2 : 1, num_sms), ns = gemv_slices(B, a.K, rpc, NORM != 0);
    const size_t smem = gemv_smem_bytes(B, a.K, rpc, ns);
    if (smem > gemv_most(NORM != 0)) return -1000;
    static SmemOptIn seen;
    if (const int e = ensure_dyn_smem(gemv_kernel<B, EPI, NORM>, smem, seen)) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(num_sms);
    cfg.blockDim = dim3(GV_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return (int)cudaLaunchKernelEx(&cfg, gemv_kernel<B, EPI, NORM>, a, ns);
}

template <int B>
static int gemv_launch_b(cudaStream_t st, int epi, bool norm, const GemvArgs& a, int num_sms, bool pdl) {
    if (norm && a.fs_x) {
        if (a.fs_n < 1 || a.fs_n > 4 || a.fs_x == a.fs_next) return -1000;
        return epi == GEMV_STORE ? gemv_launch_t<B, GEMV_STORE, 2>(st, a, num_sms, pdl) : epi == GEMV_RELU2 ? gemv_launch_t<B, GEMV_RELU2, 2>(st, a, num_sms, pdl) : -1000;
    }
    switch (epi) {
        case GEMV_STORE:
            return norm ? gemv_launch_t<B, GEMV_STORE, 1>(st, a, num_sms, pdl) : gemv_launch_t<B, GEMV_STORE, 0>(st, a, num_sms, pdl);
        case GEMV_RESID: return gemv_launch_t<B, GEMV_RESID, 0>(st, a, num_sms, pdl);
        case GEMV_RELU2: return norm ? -1000 : gemv_launch_t<B, GEMV_RELU2, 0>(st, a, num_sms, pdl);
        case GEMV_SILU_MUL:
            return norm ? gemv_launch_t<B, GEMV_SILU_MUL, 1>(st, a, num_sms, pdl) : gemv_launch_t<B, GEMV_SILU_MUL, 0>(st, a, num_sms, pdl);
        case GEMV_LOGITS_ARGMAX: return gemv_launch_t<B, GEMV_LOGITS_ARGMAX, 1>(st, a, num_sms, pdl);
        default: return -1000;
    }
}

// Largest sequence group (4, 2 or 1) whose f32 activations fit next to the weight rings for an in_dim of K.
int gemv_max_group(int K, int N, int num_sms) {
    for (int B : {4, 2})
        if (gemv_smem_bytes(B, K, gemv_rpc(N, 1, num_sms), 1) <= gemv_most(true)) return B;
    return 1;
}

int gemv_launch(cudaStream_t st, int B, int epi, bool norm, const GemvArgs& a, int num_sms, bool pdl) {
    if ((a.K % 256) != 0 || a.N <= 0) return -1000;      // a 512-byte chunk must not straddle rows
    if (epi == GEMV_SILU_MUL && (a.N % 2) != 0) return -1000;
    switch (B) {
        case 1: return gemv_launch_b<1>(st, epi, norm, a, num_sms, pdl);
        case 2: return gemv_launch_b<2>(st, epi, norm, a, num_sms, pdl);
        case 4: return gemv_launch_b<4>(st, epi, norm, a, num_sms, pdl);
        default: return -1000;
    }
}

// =====================================================================================
// Next-token embedding gather for the host-driven path (token id arrives from the host)
// =====================================================================================
__global__ void __launch_bounds__(256)
embed_decode_kernel(const bf16* __restrict__ embed, int H, const SeqState* __restrict__ state, float* __restrict__ x) {
    pdl_wait();
    pdl_launch_dependents();
    const int b = blockIdx.x;
    const bf16* row = embed + (size_t)state[b].token * H;
    for (int i = threadIdx.x; i < H; i += blockDim.x) x[(size_t)b * H + i] = __bfloat162float(row[i]);
}

__global__ void __launch_bounds__(SEQ_PACK)
set_state_kernel(SeqState* __restrict__ state, const __grid_constant__ SeqPack pack, int n) {
    pdl_launch_dependents();
    if ((int)threadIdx.x < n) state[threadIdx.x] = pack.s[threadIdx.x];
}
int set_state_launch(cudaStream_t st, SeqState* state, const SeqState* snapshots, int n) {
    if (n < 1 || n > SEQ_PACK) return -1000;
    SeqPack pack = {};
    for (int i = 0; i < n; ++i) pack.s[i] = snapshots[i];
    return launch_k(set_state_kernel, dim3(1), dim3(SEQ_PACK), 0, st, false, state, pack, n);
}

// blockIdx.y: segment.  Bound by HBM for long segments (four 16-byte loads in flight per thread), by the launch for short ones.
__global__ void __launch_bounds__(256)
copy_list_kernel(const __grid_constant__ CopyList list) {
    const CopySeg g = list.s[blockIdx.y];
    const size_t n = g.bytes / 16, step = (size_t)gridDim.x * 256;
    uint4* d = reinterpret_cast<uint4*>(g.dst);
    const uint4* s = reinterpret_cast<const uint4*>(g.src);
    uint4* k = reinterpret_cast<uint4*>(g.park);
    for (size_t i = blockIdx.x * (size_t)256 + threadIdx.x; i < n; i += 4 * step) {
        uint4 v[4], o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (i + j * step < n) { v[j] = s ? s[i + j * step] : make_uint4(0u, 0u, 0u, 0u); if (k) o[j] = d[i + j * step]; }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (i + j * step < n) { if (k) k[i + j * step] = o[j]; d[i + j * step] = v[j]; }
    }
}
int copy_list_launch(cudaStream_t st, const CopyList& list) {
    if (list.n < 0 || list.n > COPY_LIST) return -1000;
    if (list.n == 0) return 0;
    size_t most = 0;
    for (int i = 0; i < list.n; ++i) most = std::max(most, list.s[i].bytes);
    const size_t blocks = (most / 16 + 1023) / 1024;
    copy_list_kernel<<<dim3((unsigned)std::max<size_t>(1, std::min<size_t>(blocks, 64)), list.n), 256, 0, st>>>(list);
    return (int)cudaGetLastError();
}

// =====================================================================================
// Greedy argmax of a batch's logits rows (two launches: parts of every row, then one block per row)
// =====================================================================================
__device__ __forceinline__ void arg_better(float& bv, int& bi, float v, int i) {
    if (v > bv || (v == bv && i < bi)) { bv = v; bi = i; }
}
__device__ __forceinline__ void arg_warp(float& bv, int& bi) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        arg_better(bv, bi, ov, oi);
    }
}
__global__ void __launch_bounds__(256)
argmax_row_parts_kernel(const float* __restrict__ logits, int V, float* __restrict__ pv, int* __restrict__ pi) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ float sv[8];
    __shared__ int si[8];
    const int b = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float* row = logits + (size_t)b * V;
    const int per = (V + ARGMAX_ROW_PARTS - 1) / ARGMAX_ROW_PARTS, lo = blockIdx.x * per, hi = min(V, lo + per);
    float bv = -INFINITY; int bi = 0x7fffffff;
    for (int i = lo + threadIdx.x; i < hi; i += 256) if (row[i] > bv) { bv = row[i]; bi = i; }
    arg_warp(bv, bi);
    if (lane == 0) { sv[warp] = bv; si[warp] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) arg_better(bv, bi, sv[w], si[w]);
        pv[b * ARGMAX_ROW_PARTS + blockIdx.x] = bv; pi[b * ARGMAX_ROW_PARTS + blockIdx.x] = bi;
    }
}
__global__ void __launch_bounds__(256)
argmax_row_finish_kernel(const float* __restrict__ pv, const int* __restrict__ pi, SeqState* state, uint32_t* out_tokens, int out_stride,
                         const bf16* __restrict__ embed, float* __restrict__ x_next, int H, int V, int advance) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ uint32_t tok_s;
    const int b = blockIdx.x;
    if (threadIdx.x < 32) {
        float bv = pv[b * ARGMAX_ROW_PARTS + threadIdx.x]; int bi = pi[b * ARGMAX_ROW_PARTS + threadIdx.x];
        arg_warp(bv, bi);
        if ((unsigned)bi >= (unsigned)V) bi = 0;             // an all-NaN row has no maximum: never gather from an out-of-range id
        if (threadIdx.x == 0) {
            SeqState* s = state + b;
            out_tokens[(size_t)b * out_stride + s->step] = (uint32_t)bi;
            const uint32_t fed = advance == 2 ? s->token : (uint32_t)bi;
            tok_s = fed;
            if (advance) { s->token = fed; s->kv_len += 1; s->pos[0] += 1; s->pos[1] += 1; s->pos[2] += 1; }
            s->step += 1;
        }
    }
    __syncthreads();
    if (advance && embed != nullptr) {
        const bf16* row = embed + (size_t)tok_s * H;
        for (int i = threadIdx.x; i < H; i += 256) x_next[(size_t)b * H + i] = __bfloat162float(row[i]);
    }
}
int argmax_rows_launch(cudaStream_t st, int B, const float* logits, int V, float* part_val, int* part_idx, SeqState* state, uint32_t* out_tokens, int out_stride,
                       const bf16* embed, float* x_next, int H, int advance, bool pdl) {
    if (const int e = launch_k(argmax_row_parts_kernel, dim3(ARGMAX_ROW_PARTS, B), dim3(256), 0, st, pdl, logits, V, part_val, part_idx)) return e;
    return launch_k(argmax_row_finish_kernel, dim3(B), dim3(256), 0, st, pdl, part_val, part_idx, state, out_tokens, out_stride, embed, x_next, H, V, advance);
}

int embed_decode_launch(cudaStream_t st, int B, const bf16* embed, int H, const SeqState* state, float* x, bool pdl) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(B);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return (int)cudaLaunchKernelEx(&cfg, embed_decode_kernel, embed, H, state, x);
}

// =====================================================================================
// Decode attention: QK-norm + (M)RoPE + KV-page append + split-KV GQA attention + in-cluster split merge
//   grid (nkv * nsplit, B), 256 threads, thread-block CLUSTER of nsplit (1 .. 8) CTAs per KV head and sequence.
//   * the K/V rows are requested BEFORE griddepcontrol.wait: cached K/V and the sequence state were written at least two kernels ago,
//     so (the first part of) the KV read overlaps the QKV linear that precedes this kernel;
//   * RING (bf16 pages): every lane streams its own 16-byte pieces through a private ring of ATTN_DEPTH places -- it copies what it
//     reads itself, so nothing but its own copies is waited for -- and 96 KB per CTA keep two CTAs on an SM.  (Tiles of 128 KB shared by the CTA,
//     one CTA per SM, load and compute in turn: 171 us for 32 sequences of 135 .. 900 tokens, 8 KV heads; the bytes take 23.)
//     Quantised pages are dequantised into shared tiles instead;
//   * all NREP query heads of the KV group share every K/V byte (read once per group, 16-byte vectors);
//   * the split partials are merged through distributed shared memory (no global round trip, no atomics).
// =====================================================================================
constexpr int ATTN_DEPTH = 6;

template <int D, int NREP, bool RING>
__global__ void __launch_bounds__(256)
attn_decode_kernel(AttnDecArgs a) {
    namespace cg = cooperative_groups;
    constexpr int EPL = 8;               // bf16 elements per 16-byte lane load
    constexpr int LPT = D / EPL;         // lanes per token (16 for D=128, 32 for D=256)
    constexpr int TPW = 32 / LPT;        // tokens per warp pass
    constexpr int NW = 8;
    static_assert(NREP < NW, "one q/k vector per warp");
    constexpr int TILE = 32768 / (D * 2);   // tokens per shared-memory tile (K and V: 32 KB each)
    constexpr int CPR = D / 8;              // 16-byte chunks per token row
    extern __shared__ __align__(16) unsigned char asm_[];
    bf16* k_t = reinterpret_cast<bf16*>(asm_);
    bf16* v_t = k_t + TILE * D;
    bf16* kl_t = v_t + TILE * D;          // split precision only: low-order planes of the same tile
    bf16* vl_t = kl_t + TILE * D;
    const bool split_kv = a.kv_bits ? (a.kv_split != 0) : (a.kv_lo_off != 0);
    float* mo_s = reinterpret_cast<float*>(asm_);          // [NW][NREP][D], aliases the tiles after the token loop
    __shared__ float q_s[NREP][D];
    __shared__ float knew_s[D], vnew_s[D];
    __shared__ float mm_s[NW][NREP], ml_s[NW][NREP];
    __shared__ float part_o[NREP * D + ATTN_NSPLIT];         // [split][this CTA's share of the outputs], written by the cluster's CTAs
    __shared__ float part_ml[ATTN_NSPLIT][NREP][2];

    cg::cluster_group cluster = cg::this_cluster();
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");      // (waited for before the first write to another CTA's shared memory)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // a KV head whose query group is wider than NREP is served by `groups` CTA clusters of NREP query heads each (6 = 2 x 3,
    // 8 = 2 x 4, ...): kvv numbers those sub-groups, query head = kvv * NREP + h; only sub-group 0 appends the new K/V row
    const int ns = RING ? a.nsplit : ATTN_NSPLIT, kvv = blockIdx.x / ns, split = blockIdx.x % ns;
    const int kvh = kvv / a.groups, sub = kvv % a.groups;
    const int b = blockIdx.y;
    const int q_dim = a.nh * D, kv_dim = a.nkv * D;
    const int q_span = a.nh * a.q_stride;

    // ---- token range of this split, then start the K/V copy (independent of the previous kernel) ----
    const SeqState st = a.state[b];
    const int T = st.kv_len + 1;                      // including the token being decoded
    int chunk = (T + ns - 1) / ns;
    chunk = (chunk + 7) & ~7;
    const int t0 = split * chunk;
    const int t1 = min(T, t0 + chunk);
    const int s_last = (T - 1) / chunk;
    const int t_end = min(t1, T - 1);                 // cached tokens only; position T-1 comes from this step's qkv
    const int* bt = a.block_table + (size_t)st.slot * a.max_pages;
    auto load_tile = [&](int tb) {
        const int n = min(TILE, t_end - tb);
        if (a.kv_bits) {
            // codes -> (code - offset) * scale -> bf16 hi (+ lo) rows of the tile: 16 elements per thread and pass
            const int off = a.kv_bits == 8 ? 128 : 8;
            for (int c = tid; c < n * (D / 16) * 2; c += 256) {
                const int which = c & 1, cc = c >> 1;
                const int r = cc / (D / 16), ch = cc % (D / 16);
                const int t = tb + r;
                const size_t prow = ((size_t)bt[t / KV_PAGE] * a.nkv + kvh) * KV_PAGE + (t % KV_PAGE);
                const unsigned char* codes = which ? a.v_codes : a.k_codes;
                const float scale = (which ? a.v_scale : a.k_scale)[prow];
                int q[16];
                if (a.kv_bits == 8) {
                    const uint4 u = *reinterpret_cast<const uint4*>(codes + prow * D + ch * 16);
                    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                    for (int e = 0; e < 16; ++e) q[e] = (int)((w[e >> 2] >> (8 * (e & 3))) & 255u);
                } else {
                    const uint2 u = *reinterpret_cast<const uint2*>(codes + prow * (D / 2) + ch * 8);
                    const uint32_t w[2] = {u.x, u.y};
#pragma unroll
                    for (int e = 0; e < 16; ++e) q[e] = (int)((w[e >> 3] >> (4 * (e & 7))) & 15u);
                }
                bf16* hi_t = (which ? v_t : k_t) + r * D + ch * 16;
                bf16* lo_t = (which ? vl_t : kl_t) + r * D + ch * 16;
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const float y = (float)(q[e] - off) * scale;
                    const bf16 hb = __float2bfloat16_rn(y);
                    hi_t[e] = hb;
                    if (split_kv) lo_t[e] = __float2bfloat16_rn(y - __bfloat162float(hb));
                }
            }
            return;
        }
        for (int c = tid; c < n * CPR; c += 256) {
            const int r = c / CPR, ch = c % CPR;
            const int t = tb + r;
            const int page = bt[t / KV_PAGE];
            const size_t off = (((size_t)page * a.nkv + kvh) * KV_PAGE + (t % KV_PAGE)) * D + ch * 8;
            const uint32_t kd = smem_u32(k_t + r * D + ch * 8), vd = smem_u32(v_t + r * D + ch * 8);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(kd), "l"(a.k_pool + off) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(vd), "l"(a.v_pool + off) : "memory");
            if (split_kv) {
                const uint32_t kld = smem_u32(kl_t + r * D + ch * 8), vld = smem_u32(vl_t + r * D + ch * 8);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(kld), "l"(a.k_pool + a.kv_lo_off + off) : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(vld), "l"(a.v_pool + a.kv_lo_off + off) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // RING: token groups r0 = t0 + warp * TPW + i * NW * TPW of this warp; a lane's place holds its pieces of K hi, V hi, K lo, V lo, 512 bytes apart
    const int grp = lane / LPT, gl = lane % LPT;        // token group inside the warp, lane inside the group
    const int w0 = t0 + warp * TPW, n_it = max(0, (t_end - w0 + NW * TPW - 1) / (NW * TPW));
    unsigned char* ring = asm_ + (size_t)warp * ATTN_DEPTH * 2048 + lane * 16;
    const uint32_t ring_u32 = smem_u32(ring);
    auto ring_issue = [&](int i) {
        const int t = w0 + i * NW * TPW + grp;
        if (i < n_it && t < t_end) {
            const size_t off = (((size_t)bt[t / KV_PAGE] * a.nkv + kvh) * KV_PAGE + (t % KV_PAGE)) * D + gl * EPL;
            const uint32_t dst = ring_u32 + (uint32_t)(i % ATTN_DEPTH) * 2048;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(a.k_pool + off) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 512), "l"(a.v_pool + off) : "memory");
            if (split_kv) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 1024), "l"(a.k_pool + a.kv_lo_off + off) : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 1536), "l"(a.v_pool + a.kv_lo_off + off) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if constexpr (RING) {
#pragma unroll
        for (int i = 0; i < ATTN_DEPTH; ++i) ring_issue(i);
    } else {
        if (t0 < t_end) load_tile(t0);
    }

    // norm weights and this position's cos/sin depend only on immutable data and the sequence state: fetch them before
    // the dependency wait too (lane l owns elements l + 32 j, so a rotary pair is lane-local)
    constexpr int NE = D / 32;
    const int RJ = a.rot_half >> 5;                    // lane-local rotary pairs (j, j + RJ), j < RJ
    const bool vec_is_k = (warp == NREP);
    float nwv[NE], cs_c[NE], cs_s[NE];
    if (warp <= NREP) {
        const float* nw = vec_is_k ? a.k_norm_w : a.q_norm_w;
#pragma unroll
        for (int j = 0; j < NE; ++j) {
            nwv[j] = nw[lane + 32 * j];
            cs_c[j] = 1.f; cs_s[j] = 0.f;
            if (j < 2 * RJ) {
                const int i = lane + 32 * (j < RJ ? j : j - RJ);
                const int p = st.pos[a.axis_of[i]];
                cs_c[j] = a.cos_tab[(size_t)p * a.rot_half + i];
                cs_s[j] = a.sin_tab[(size_t)p * a.rot_half + i];
            }
        }
    }

    pdl_wait();
    pdl_launch_dependents();
    const float* qkv = a.qkv + (size_t)b * (q_span + 2 * kv_dim);

    // ---- q (NREP heads) and, on the split that owns position T-1, the new k: RMSNorm then rotate ----
    for (int vec = warp; vec < NREP + 1; vec += NW) {      // NW > NREP: one vector per warp, vec == warp
        const bool is_k = (vec == NREP);
        if (is_k && split != s_last) continue;
        const float* src = is_k ? (qkv + q_span + kvh * D) : (qkv + (kvv * NREP + vec) * a.q_stride);
        float e[NE];
        float ssq = 0.f;
#pragma unroll
        for (int j = 0; j < NE; ++j) { e[j] = src[lane + 32 * j]; ssq += e[j] * e[j]; }
        ssq = warp_sum(ssq);
        const float rstd = rsqrtf(ssq / (float)D + a.eps);
#pragma unroll
        for (int j = 0; j < NE; ++j) e[j] = e[j] * rstd * nwv[j];
        float* dst = is_k ? knew_s : q_s[vec];
#pragma unroll
        for (int j = 0; j < NE; ++j) {
            float r = e[j];
            if (j < 2 * RJ) {
                const bool lo = j < RJ;
                const float c = cs_c[j], s = cs_s[j];
                float other = 0.f;
#pragma unroll
                for (int jj = 0; jj < NE; ++jj) if (jj == (lo ? j + RJ : j - RJ)) other = e[jj];
                r = lo ? (e[j] * c - other * s) : (other * s + e[j] * c);
            }
            dst[lane + 32 * j] = (is_k && !a.kv_bits) ? (split_kv ? round_bf16_split(r) : round_bf16(r)) : r;
        }
    }
    if (split == s_last && warp == NW - 1) {
        const float* vsrc = qkv + q_span + kv_dim + kvh * D;
        for (int i = lane; i < D; i += 32) vnew_s[i] = a.kv_bits ? vsrc[i] : (split_kv ? round_bf16_split(vsrc[i]) : round_bf16(vsrc[i]));
    }
    __syncthreads();
    if (a.kv_bits && split == s_last && warp < 2) {
        // quantise the new K (warp 0) / V (warp 1) row per token and head; attention -- here and in every later step -- sees code * scale
        float* row = warp ? vnew_s : knew_s;
        const int t = T - 1;
        const size_t prow = ((size_t)bt[t / KV_PAGE] * a.nkv + kvh) * KV_PAGE + (t % KV_PAGE);
        float am = 0.f;
        for (int i = lane; i < D; i += 32) am = fmaxf(am, fabsf(row[i]));
        am = warp_max(am);
        const float inv = a.kv_bits == 8 ? (float)(1.0 / 127.0) : (float)(1.0 / 7.0);
        const float scale = __fadd_rn(__fmul_rn(am, inv), 1e-8f);
        const int off = a.kv_bits == 8 ? 128 : 8;
        unsigned char* codes = warp ? a.v_codes : a.k_codes;
        for (int i = 2 * lane; i < D; i += 64) {          // an (even, odd) pair per lane and pass
            const int q0 = (int)roundf(__fdiv_rn(row[i], scale)), q1 = (int)roundf(__fdiv_rn(row[i + 1], scale));
            row[i] = (float)q0 * scale; row[i + 1] = (float)q1 * scale;
            if (sub == 0) {
                if (a.kv_bits == 8) { codes[prow * D + i] = (unsigned char)(q0 + off); codes[prow * D + i + 1] = (unsigned char)(q1 + off); }
                else codes[prow * (D / 2) + (i >> 1)] = (unsigned char)((q0 + off) + 16 * (q1 + off));
            }
        }
        if (sub == 0 && lane == 0) (warp ? a.v_scale : a.k_scale)[prow] = scale;
    }
    if (a.kv_bits) __syncthreads();
    if (!a.kv_bits && split == s_last && sub == 0) {   // append the new token to its page
        const int t = T - 1;
        const int page = bt[t / KV_PAGE];
        const size_t off = (((size_t)page * a.nkv + kvh) * KV_PAGE + (t % KV_PAGE)) * D;
        for (int i = tid; i < D; i += 256) {
            const bf16 kh = __float2bfloat16_rn(knew_s[i]), vh = __float2bfloat16_rn(vnew_s[i]);
            a.k_pool[off + i] = kh;
            a.v_pool[off + i] = vh;
            if (split_kv) {
                a.k_pool[a.kv_lo_off + off + i] = __float2bfloat16_rn(knew_s[i] - __bfloat162float(kh));
                a.v_pool[a.kv_lo_off + off + i] = __float2bfloat16_rn(vnew_s[i] - __bfloat162float(vh));
            }
        }
    }

    // ---- the cached tokens of this split, tile by tile out of shared memory ----
    float qr[NREP][EPL];
#pragma unroll
    for (int h = 0; h < NREP; ++h)
#pragma unroll
        for (int j = 0; j < EPL; ++j) qr[h][j] = q_s[h][gl * EPL + j] * a.scale;
    float m[NREP], l[NREP], o[NREP][EPL];
#pragma unroll
    for (int h = 0; h < NREP; ++h) {
        m[h] = -INFINITY; l[h] = 0.f;
#pragma unroll
        for (int j = 0; j < EPL; ++j) o[h][j] = 0.f;
    }
    // U tokens of this lane's group at a time: their scores, shuffles and exponentials are independent, where token by token they were a chain of five dependent
    // steps.  The running sums take them one after the other all the same: rescaled once for both they were rounded otherwise, and what a quantised model's codes
    // make of that is 1e-2 of its logits.  (32 sequences of 45 .. 300 tokens, 32 heads over 8 of D = 128: 30.1 us, 34.1 token by token, 28.9 rescaled once.)
    constexpr int U = 2;
    auto unpack = [&](float* f, const bf16* hp, const bf16* lp) __attribute__((always_inline)) {
        const uint4 r = *reinterpret_cast<const uint4*>(hp);
        f[0] = bf16lo(r.x); f[1] = bf16hi(r.x); f[2] = bf16lo(r.y); f[3] = bf16hi(r.y);
        f[4] = bf16lo(r.z); f[5] = bf16hi(r.z); f[6] = bf16lo(r.w); f[7] = bf16hi(r.w);
        if (split_kv) {
            const uint4 q = *reinterpret_cast<const uint4*>(lp);
            f[0] += bf16lo(q.x); f[1] += bf16hi(q.x); f[2] += bf16lo(q.y); f[3] += bf16hi(q.y);
            f[4] += bf16lo(q.z); f[5] += bf16hi(q.z); f[6] += bf16lo(q.w); f[7] += bf16hi(q.w);
        }
    };
    auto attend = [&](const bool* valid, const bf16* const* kp, const bf16* const* vp, int lo) __attribute__((always_inline)) {
        float sc[U][NREP];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float kf[EPL];
#pragma unroll
            for (int j = 0; j < EPL; ++j) kf[j] = 0.f;
            if (valid[u]) unpack(kf, kp[u], kp[u] + lo);
#pragma unroll
            for (int h = 0; h < NREP; ++h) {
                float s = 0.f;
#pragma unroll
                for (int j = 0; j < EPL; ++j) s = fmaf(qr[h][j], kf[j], s);
                sc[u][h] = s;
            }
        }
#pragma unroll
        for (int ofs = LPT / 2; ofs > 0; ofs >>= 1)
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int h = 0; h < NREP; ++h) sc[u][h] += __shfl_xor_sync(0xffffffffu, sc[u][h], ofs);
        if (!valid[0]) return;                          // (tokens ascend: the others are not there either)
        float c[U][NREP];
#pragma unroll
        for (int h = 0; h < NREP; ++h)
#pragma unroll
            for (int u = 0; u < U; ++u) {               // (a token that is not there: factor 1, weight 0)
                const float mn = valid[u] ? fmaxf(m[h], sc[u][h]) : m[h];
                c[u][h] = __expf(m[h] - mn);
                sc[u][h] = valid[u] ? __expf(sc[u][h] - mn) : 0.f;
                l[h] = l[h] * c[u][h] + sc[u][h];
                m[h] = mn;
            }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float vf[EPL];
#pragma unroll
            for (int j = 0; j < EPL; ++j) vf[j] = 0.f;
            if (valid[u]) unpack(vf, vp[u], vp[u] + lo);
#pragma unroll
            for (int h = 0; h < NREP; ++h)
#pragma unroll
                for (int j = 0; j < EPL; ++j) o[h][j] = o[h][j] * c[u][h] + sc[u][h] * vf[j];
        }
    };
    bool valid[U];
    const bf16 *kp[U], *vp[U];
    if constexpr (RING) {
        static_assert(ATTN_DEPTH % U == 0, "a turn's slots are neighbours");
        for (int i = 0; i < n_it; i += U) {
            asm volatile("cp.async.wait_group %0;" ::"n"(ATTN_DEPTH - U) : "memory");
#pragma unroll
            for (int u = 0; u < U; ++u) {
                valid[u] = w0 + (i + u) * NW * TPW + grp < t_end;
                kp[u] = reinterpret_cast<const bf16*>(ring + ((i + u) % ATTN_DEPTH) * 2048); vp[u] = kp[u] + 256;
            }
            attend(valid, kp, vp, 512);
#pragma unroll
            for (int u = 0; u < U; ++u) ring_issue(i + u + ATTN_DEPTH);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else {
        for (int tb = t0; tb < t_end; tb += TILE) {
            if (tb != t0) { __syncthreads(); load_tile(tb); }
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            const int n = min(TILE, t_end - tb);
            for (int r0 = warp * TPW; r0 < n; r0 += U * NW * TPW) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int r = r0 + u * NW * TPW + grp, o_ = r * D + gl * EPL;
                    valid[u] = r < n; kp[u] = k_t + o_; vp[u] = v_t + o_;
                }
                attend(valid, kp, vp, 2 * TILE * D);
            }
        }
    }
    // the token being decoded (K/V still in shared memory): group 0 of warp 0 on the owning split
    if (split == s_last && warp == 0 && grp == 0) {
#pragma unroll
        for (int h = 0; h < NREP; ++h) {
            float s = 0.f;
#pragma unroll
            for (int j = 0; j < EPL; ++j) s = fmaf(qr[h][j], knew_s[gl * EPL + j], s);
#pragma unroll
            for (int ofs = LPT / 2; ofs > 0; ofs >>= 1) s += __shfl_xor_sync((TPW == 1) ? 0xffffffffu : 0x0000ffffu, s, ofs);
            const float mn = fmaxf(m[h], s);
            const float corr = __expf(m[h] - mn), p = __expf(s - mn);
            l[h] = l[h] * corr + p;
#pragma unroll
            for (int j = 0; j < EPL; ++j) o[h][j] = o[h][j] * corr + p * vnew_s[gl * EPL + j];
            m[h] = mn;
        }
    }
    // merge the token groups of a warp
    if (TPW == 2) {
#pragma unroll
        for (int h = 0; h < NREP; ++h) {
            const float mo = __shfl_xor_sync(0xffffffffu, m[h], 16);
            const float lo = __shfl_xor_sync(0xffffffffu, l[h], 16);
            const float mn = fmaxf(m[h], mo);
            const float c0 = (m[h] == -INFINITY) ? 0.f : __expf(m[h] - mn);
            const float c1 = (mo == -INFINITY) ? 0.f : __expf(mo - mn);
            l[h] = l[h] * c0 + lo * c1;
#pragma unroll
            for (int j = 0; j < EPL; ++j) {
                const float oo = __shfl_xor_sync(0xffffffffu, o[h][j], 16);
                o[h][j] = o[h][j] * c0 + oo * c1;
            }
            m[h] = mn;
        }
    }
    __syncthreads();                                     // tiles are dead: reuse them as the warp-merge buffer
    if (grp == 0) {
#pragma unroll
        for (int h = 0; h < NREP; ++h) {
            if (gl == 0) { mm_s[warp][h] = m[h]; ml_s[warp][h] = l[h]; }
#pragma unroll
            for (int j = 0; j < EPL; ++j) mo_s[((size_t)warp * NREP + h) * D + gl * EPL + j] = o[h][j];
        }
    }
    __syncthreads();
    // merge the warps, and push the result to the CTAs that merge the splits: CTA r of the cluster finishes outputs [r * per, (r + 1) * per).  Written to where
    // they are read, the partials take one barrier; read from where they were made they took two round trips and a second barrier (1 sequence of
    // 128 tokens, D = 128: 4.6 us a launch among its like, 5.3 before).
    constexpr int E = NREP * D;
    const int per = (E + ns - 1) / ns;
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");        // every CTA of the cluster runs
    for (int idx = tid; idx < E; idx += 256) {
        const int h = idx / D, i = idx % D;
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < NW; ++w) M = fmaxf(M, mm_s[w][h]);
        float L = 0.f, O = 0.f;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            const float c = (mm_s[w][h] == -INFINITY) ? 0.f : __expf(mm_s[w][h] - M);
            L += ml_s[w][h] * c;
            O += mo_s[((size_t)w * NREP + h) * D + i] * c;
        }
        const int to = idx / per;
        *cluster.map_shared_rank(&part_o[split * per + (idx - to * per)], to) = O;
        if (i < ns) {                                    // (ns <= 8 < D: lane i of a head tells CTA i)
            float* ml = cluster.map_shared_rank(&part_ml[split][h][0], i);
            ml[0] = M; ml[1] = L;
        }
    }
    cluster.sync();
    for (int t = tid; t < per && split * per + t < E; t += 256) {
        const int idx = split * per + t, h = idx / D, i = idx % D;
        float M = -INFINITY;
#pragma unroll
        for (int s = 0; s < ATTN_NSPLIT; ++s) if (!RING || s < ns) M = fmaxf(M, part_ml[s][h][0]);
        float L = 0.f, O = 0.f;
#pragma unroll
        for (int s = 0; s < ATTN_NSPLIT; ++s)
            if (!RING || s < ns) {
                const float ms = part_ml[s][h][0], c = (ms == -INFINITY) ? 0.f : __expf(ms - M);
                L += part_ml[s][h][1] * c;
                O += part_o[s * per + t] * c;
            }
        const int head = kvv * NREP + h;
        float r = O / L;
        if (a.gated) r *= 1.0f / (1.0f + expf(-qkv[head * a.q_stride + D + i]));   // y * sigmoid(gate), modeling.rs:516-523
        a.out[(size_t)b * q_dim + head * D + i] = r;
    }
}

template <int D, int NREP, bool RING>
static int attn_decode_launch_t(cudaStream_t st, int B, const AttnDecArgs& a, bool pdl) {
    const int SMEM = RING ? 8 * ATTN_DEPTH * 2048 : (a.kv_bits ? a.kv_split : (a.kv_lo_off != 0)) ? 131072 : 65536;
    static SmemOptIn seen;
    if (const int e = ensure_dyn_smem(attn_decode_kernel<D, NREP, RING>, (size_t)SMEM, seen)) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.nkv * a.groups * a.nsplit, B);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = a.nsplit; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 2 : 1;
    return (int)cudaLaunchKernelEx(&cfg, attn_decode_kernel<D, NREP, RING>, a);
}
// Tile form (a CTA requests its whole range ahead of the dependency wait) while its clusters of eight, one per (sequence, KV group), run at once: in split
// precision a tile takes an SM, in plain bf16 a third of one.  Rings beyond.  us, tile / rings, contexts of 1000 tokens, single launches with cold caches (C: clusters):
//   split, D = 128   2 KV heads of 2: 3 sequences (12 C) 10.1 / 10.5, 6 (12 C) 11.7 / 12.0, 9 (18 C) 19.6 / 13.7     4 heads: 3 (12 C) 11.9 / 12.7, 4 (16 C) 19.5 / 13.5
//                    8 KV heads: 2 sequences (16 C) 19.0 / 13.1, 4 28.2 / 15.1
//   split, D = 256   2 KV heads: 1 sequence 15.7 / 15.5, 5 (10 C) 18.0 / 17.7, 8 (16 C) 31.6 / 20.6     8 heads: 1 16.9 / 17.3, 2 (16 C) 31.6 / 20.9
//   plain, D = 128   8 KV heads: 4 sequences (32 C) 12.4 / 12.8, 5 (40 C) 15.0 / 16.3; 64 heads over 8: 2 (32 C) 15.6 / 16.0, 3 (48 C) 26.2 / 21.4
//   plain, D = 256   2 KV heads: 8 sequences 18.0 / 18.4; 8 heads: 4 (32 C) 19.8 / 19.7
static bool attn_tile_form(const AttnDecArgs& a, int pairs) { return a.kv_bits || pairs <= (a.kv_lo_off ? tc_max_clusters(ATTN_NSPLIT) : 32); }

template <int D, int NREP>
static int attn_decode_launch_r(cudaStream_t st, int B, const AttnDecArgs& a, bool pdl) {
    return attn_tile_form(a, B * a.nkv * a.groups) ? attn_decode_launch_t<D, NREP, false>(st, B, a, pdl) : attn_decode_launch_t<D, NREP, true>(st, B, a, pdl);
}

int attn_decode_launch(cudaStream_t st, int B, int D, const AttnDecArgs& a_in, bool pdl) {
    AttnDecArgs a = a_in;
    if (a.nkv <= 0 || a.nh <= 0 || a.nh % a.nkv) return -1000;
    const int nrep = a.nh / a.nkv;
    if (a.rot_half < 32 || (a.rot_half % 32) != 0 || 2 * a.rot_half > D) return -1000;
    // any group width: the widest instantiated sub-group (4, 3, 2, 1 query heads) that divides it
    int sub = nrep % 4 == 0 ? 4 : nrep % 3 == 0 ? 3 : nrep % 2 == 0 ? 2 : 1;
    // narrower ones while all their clusters still run at once: few clusters leave most of the chip idle, and a CTA's time goes with its heads, not with the
    // bytes the sub-groups read again (1 sequence, 8 heads over 2 of D = 256: 1000 tokens 9.4 us, 12.2 before)
    while (sub % 2 == 0 && B * a.nkv * (nrep / sub * 2) <= tc_max_clusters(ATTN_NSPLIT)) sub /= 2;
    a.groups = nrep / sub;
    // splits per (sequence, KV group): all eight while they leave SMs idle, fewer as the batch itself fills the chip (two CTAs per SM)
    const int pairs = B * a.nkv * a.groups;
    a.nsplit = pairs <= 37 ? 8 : pairs <= 148 ? 4 : pairs <= 512 ? 2 : 1;
    if (attn_tile_form(a, pairs)) a.nsplit = ATTN_NSPLIT;      // (its split is fixed)
    if (D == 128) {
        switch (sub) {
            case 1: return attn_decode_launch_r<128, 1>(st, B, a, pdl);
            case 2: return attn_decode_launch_r<128, 2>(st, B, a, pdl);
            case 3: return attn_decode_launch_r<128, 3>(st, B, a, pdl);
            case 4: return attn_decode_launch_r<128, 4>(st, B, a, pdl);
        }
    } else if (D == 256) {
        switch (sub) {
            case 1: return attn_decode_launch_r<256, 1>(st, B, a, pdl);
            case 2: return attn_decode_launch_r<256, 2>(st, B, a, pdl);
            case 3: return attn_decode_launch_r<256, 3>(st, B, a, pdl);
            case 4: return attn_decode_launch_r<256, 4>(st, B, a, pdl);
        }
    }
    return -1000;
}

}  // namespace cb
