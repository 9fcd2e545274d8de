// GGUF-quantised linears on the decode path: stream the QUANTISED bytes (0.56 / 0.875 / 1.06 B per weight) and do the
// dot products with dp4a on int8 activations, dequantising per block in registers -- never materialising bf16 weights.
//
// Replaces candle's `QMatMul::forward` behind `LinearLayer::Quantized` (crane-core/src/ops/linear.rs:23-48) /
// `Gguf::linear` (crane-core/src/models/hunyuan_dense/modeling.rs:37-41).  Like candle's own paths (CPU: activations
// quantised to Q8_K blocks) the activation vector is quantised to int8 blocks -- Q8_K (256 elements) in front of K-quant
// weights, Q8_0 (32 elements) in front of Q8_0 weights, with candle's own rounding rules (xquant_kernel) -- before the
// integer dot; block formats follow ggml exactly (oracle/ggml_quant.py is pinned to the `gguf` package byte for byte, and
// its `qmatmul` restates the ggml integer dots this kernel reproduces).
//
// Kernel shape is the bf16 GEMV's (decode.cu): grid = #SMs, contiguous row block per CTA, one private cp.async ring per
// warp, weights primed before griddepcontrol.wait, fused epilogues.  Two (Q4_K, Q6_K) or four (Q8_0) lanes share one
// 256-element super-block.
#include "quant.cuh"

#include <cuda_fp16.h>

#include <cstring>
#include <vector>

namespace cb {

// ------------------------------------------------------------------------------------------------ host repack
void q_repack_rows(int qt, const unsigned char* src, unsigned char* dst, size_t rows, int K) {
    const size_t nsb = (size_t)rows * (K / 256);
    if (qt == QT_Q4_K) { std::memcpy(dst, src, nsb * 144); return; }
    if (qt == QT_Q6_K) {
        for (size_t i = 0; i < nsb; ++i) {
            const unsigned char* s = src + i * 210;
            unsigned char* d = dst + i * 224;
            std::memcpy(d, s, 208);              // ql (128) | qh (64) | scales (16) keep their offsets
            std::memcpy(d + 208, s + 208, 2);    // f16 d
            std::memset(d + 210, 0, 14);
        }
        return;
    }
    for (size_t i = 0; i < nsb; ++i) {           // Q8_0: 8 blocks of [f16 d | 32 x i8] -> [256 x i8 | 8 x f16 d]
        const unsigned char* s = src + i * 8 * 34;
        unsigned char* d = dst + i * 272;
        for (int b = 0; b < 8; ++b) {
            std::memcpy(d + 32 * b, s + 34 * b + 2, 32);
            std::memcpy(d + 256 + 2 * b, s + 34 * b, 2);
        }
    }
}

// ------------------------------------------------------------------------------------------------ device helpers
__device__ __forceinline__ float f16_bits_to_float(uint32_t h) { return __half2float(__ushort_as_half((unsigned short)h)); }
__device__ __forceinline__ int dp4a_s(int a, int b, int c) { return __dp4a(a, b, c); }

template <int QT> struct QTraits;
template <> struct QTraits<QT_Q4_K> { static constexpr int SB = 144; };
template <> struct QTraits<QT_Q6_K> { static constexpr int SB = 224; };
template <> struct QTraits<QT_Q8_0> { static constexpr int SB = 272; };

// Quantised activations in shared memory, B sequences back to back, each:
//   [K int8 | K/32 float2 {d, d * sum(q)} | K/16 i32 sum(q) per 16 elements]
// The int8 part is stored in 16-byte granules XOR-swizzled by the 128-element group index, so the 8 lanes of an LDS.128
// phase (2 super-blocks x 4 quarters) hit 8 different bank groups.
__device__ __forceinline__ int xq_swz(int byte_off) {
    const int g = byte_off >> 4;
    return ((g ^ ((g >> 3) & 7)) << 4) | (byte_off & 15);
}

// One lane's slice of the activations for a k-tile: 64 elements of one super-block, held in registers while the warp
// walks the rows of the tile (the weights are read once from shared memory, the activations once per tile).
//   Q4_K / Q8_0: quarter q = elements [64q, 64q + 64)                       -> blocks 2q, 2q + 1
//   Q6_K       : half h = q >> 1, lq = q & 1: elements 128h + 32t + 16lq + [0, 16), t = 0..3 (ggml's q1..q4 interleave)
template <int QT, int B>
struct XSlice {
    int4 q[B][4];
    float d[B][4];      // Q4_K: {d0, d0*sum0, d1, d1*sum1}; Q6_K: d of blocks 4h + t; Q8_0: {d0, d1, -, -}
    float s[B][4];      // Q6_K only: 32 * d_t * isum16_t
    __device__ __forceinline__ void load(const unsigned char* xbase, size_t xb, int K, int sbk_abs, int qq) {
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const unsigned char* xq = xbase + (size_t)b * xb;
            const float2* ds = reinterpret_cast<const float2*>(xq + K);
            const int* is16 = reinterpret_cast<const int*>(xq + K + (K / 32) * 8);
            if constexpr (QT == QT_Q6_K) {
                const int h = qq >> 1, lq = qq & 1;
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const int e = sbk_abs * 256 + 128 * h + 32 * t + 16 * lq;
                    q[b][t] = *reinterpret_cast<const int4*>(xq + xq_swz(e));
                    d[b][t] = ds[e >> 5].x;
                    s[b][t] = 32.f * d[b][t] * (float)is16[e >> 4];
                }
            } else {
                const int e = sbk_abs * 256 + 64 * qq;
#pragma unroll
                for (int t = 0; t < 4; ++t) q[b][t] = *reinterpret_cast<const int4*>(xq + xq_swz(e + 16 * t));
                const float4 v = *reinterpret_cast<const float4*>(ds + (e >> 5));
                d[b][0] = v.x; d[b][1] = v.y; d[b][2] = v.z; d[b][3] = v.w;
            }
        }
    }
};

__device__ __forceinline__ int dot16(const int4& w0, const int4& w1, const int4& x0, const int4& x1) {
    int s = 0;
    s = dp4a_s(w0.x, x0.x, s); s = dp4a_s(w0.y, x0.y, s); s = dp4a_s(w0.z, x0.z, s); s = dp4a_s(w0.w, x0.w, s);
    s = dp4a_s(w1.x, x1.x, s); s = dp4a_s(w1.y, x1.y, s); s = dp4a_s(w1.z, x1.z, s); s = dp4a_s(w1.w, x1.w, s);
    return s;
}
__device__ __forceinline__ int dot8(const int4& w, const int4& x) {
    int s = 0;
    s = dp4a_s(w.x, x.x, s); s = dp4a_s(w.y, x.y, s); s = dp4a_s(w.z, x.z, s); s = dp4a_s(w.w, x.w, s);
    return s;
}

// acc[b] += (this lane's 64 elements of super-block `sb`) . x[b]; weight bits are unpacked once for all B sequences.
template <int QT, int B>
__device__ __forceinline__ void sb_quarter_dot(const unsigned char* sb, int qq, const XSlice<QT, B>& x, float* acc) {
    if constexpr (QT == QT_Q4_K) {
        const uint4 hdr = *reinterpret_cast<const uint4*>(sb);         // f16 d | f16 dmin | 12 packed 6-bit scales / mins
        const float d = f16_bits_to_float(hdr.x & 0xffffu), dmin = f16_bits_to_float(hdr.x >> 16);
        // ggml get_scale_min_k4 for sub-blocks ja = 2q, ja + 1
        const int sh = 16 * (qq & 1);
        const uint32_t ya = hdr.y >> sh, za = hdr.z >> sh, wa = hdr.w >> sh;
        int sca, ma, scb, mb;
        if (qq < 2) {
            sca = ya & 63; ma = za & 63; scb = (ya >> 8) & 63; mb = (za >> 8) & 63;
        } else {
            sca = (wa & 0xF) | (((ya >> 6) & 3) << 4);        ma = ((wa >> 4) & 0xF) | (((za >> 6) & 3) << 4);
            scb = ((wa >> 8) & 0xF) | (((ya >> 14) & 3) << 4); mb = ((wa >> 12) & 0xF) | (((za >> 14) & 3) << 4);
        }
        const uint4* qp = reinterpret_cast<const uint4*>(sb + 16 + 32 * qq);
        const uint4 w0 = qp[0], w1 = qp[1];
        int4 lo0, lo1, hi0, hi1;
        lo0.x = w0.x & 0x0F0F0F0F; lo0.y = w0.y & 0x0F0F0F0F; lo0.z = w0.z & 0x0F0F0F0F; lo0.w = w0.w & 0x0F0F0F0F;
        lo1.x = w1.x & 0x0F0F0F0F; lo1.y = w1.y & 0x0F0F0F0F; lo1.z = w1.z & 0x0F0F0F0F; lo1.w = w1.w & 0x0F0F0F0F;
        hi0.x = (w0.x >> 4) & 0x0F0F0F0F; hi0.y = (w0.y >> 4) & 0x0F0F0F0F; hi0.z = (w0.z >> 4) & 0x0F0F0F0F; hi0.w = (w0.w >> 4) & 0x0F0F0F0F;
        hi1.x = (w1.x >> 4) & 0x0F0F0F0F; hi1.y = (w1.y >> 4) & 0x0F0F0F0F; hi1.z = (w1.z >> 4) & 0x0F0F0F0F; hi1.w = (w1.w >> 4) & 0x0F0F0F0F;
        const float dsa = d * (float)sca, dsb = d * (float)scb, dma = dmin * (float)ma, dmb = dmin * (float)mb;
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const int sa = dot16(lo0, lo1, x.q[b][0], x.q[b][1]);
            const int sb2 = dot16(hi0, hi1, x.q[b][2], x.q[b][3]);
            acc[b] += dsa * x.d[b][0] * (float)sa + dsb * x.d[b][2] * (float)sb2 - dma * x.d[b][1] - dmb * x.d[b][3];
        }
    } else if constexpr (QT == QT_Q6_K) {
        const int h = qq >> 1, lq = qq & 1;
        const float d = f16_bits_to_float(*reinterpret_cast<const unsigned short*>(sb + 208));
        const uint2 scw = *reinterpret_cast<const uint2*>(sb + 192 + 8 * h);        // 8 int8 scales of this half
        const uint4 A = *reinterpret_cast<const uint4*>(sb + 64 * h + 16 * lq);
        const uint4 Bq = *reinterpret_cast<const uint4*>(sb + 64 * h + 32 + 16 * lq);
        const uint4 Hh = *reinterpret_cast<const uint4*>(sb + 128 + 32 * h + 16 * lq);
        int4 q1, q2, q3, q4;
#define CB_Q6(c) \
        q1.c = (A.c & 0x0F0F0F0F) | ((Hh.c & 0x03030303) << 4); \
        q2.c = (Bq.c & 0x0F0F0F0F) | (((Hh.c >> 2) & 0x03030303) << 4); \
        q3.c = ((A.c >> 4) & 0x0F0F0F0F) | (((Hh.c >> 4) & 0x03030303) << 4); \
        q4.c = ((Bq.c >> 4) & 0x0F0F0F0F) | (((Hh.c >> 6) & 0x03030303) << 4);
        CB_Q6(x) CB_Q6(y) CB_Q6(z) CB_Q6(w)
#undef CB_Q6
        // scale of group t is byte 2t + lq of the half's 8 scales
        const float s1 = d * (float)(signed char)((scw.x >> (8 * lq)) & 0xff), s2 = d * (float)(signed char)((scw.x >> (16 + 8 * lq)) & 0xff);
        const float s3 = d * (float)(signed char)((scw.y >> (8 * lq)) & 0xff), s4 = d * (float)(signed char)((scw.y >> (16 + 8 * lq)) & 0xff);
#pragma unroll
        for (int b = 0; b < B; ++b)      // (q - 32) . x = q . x - 32 sum(x)
            acc[b] += s1 * (x.d[b][0] * (float)dot8(q1, x.q[b][0]) - x.s[b][0]) + s2 * (x.d[b][1] * (float)dot8(q2, x.q[b][1]) - x.s[b][1]) +
                      s3 * (x.d[b][2] * (float)dot8(q3, x.q[b][2]) - x.s[b][2]) + s4 * (x.d[b][3] * (float)dot8(q4, x.q[b][3]) - x.s[b][3]);
    } else {
        const int4* wq = reinterpret_cast<const int4*>(sb + 64 * qq);
        const int4 w0 = wq[0], w1 = wq[1], w2 = wq[2], w3 = wq[3];
        const uint32_t dd = *reinterpret_cast<const uint32_t*>(sb + 256 + 4 * qq);
        const float d0 = f16_bits_to_float(dd & 0xffffu), d1 = f16_bits_to_float(dd >> 16);
#pragma unroll
        for (int b = 0; b < B; ++b)
            acc[b] += d0 * x.d[b][0] * (float)dot16(w0, w1, x.q[b][0], x.q[b][1]) + d1 * x.d[b][2] * (float)dot16(w2, w3, x.q[b][2], x.q[b][3]);
    }
}

// Sum N per-lane values over the warp in N + log2(32/N) - 1 shuffles (recursive halving): on return every lane holds in
// v[0] the warp total of value `idx`.
template <int N>
__device__ __forceinline__ void warp_reduce_scatter(float (&v)[N], int lane, int& idx) {
    idx = 0;
    int off = 16;
#pragma unroll
    for (int n = N; n > 1; n >>= 1, off >>= 1) {
        const bool up = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < n / 2; ++i) {
            const float send = up ? v[i] : v[i + n / 2];
            const float keep = up ? v[i + n / 2] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
        if (up) idx += n / 2;
    }
    for (; off > 0; off >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
}

// ------------------------------------------------------------------------------------------------ activation quantiser
// The block rule is the one candle's CPU `QMatMul::forward` applies to the activations before its integer dots (`LinearLayer::Quantized`,
// crane-core/src/ops/linear.rs:23-48):
//   XQ_Q8_K (Q4_K / Q6_K weights): BlockQ8K::from_float -- 256 elements; max = first element of largest magnitude, sign kept;
//                                  iscale = -128 / max; q = min(127, round(iscale * x)); d = 1 / iscale
//   XQ_Q8_0 (Q8_0 weights)       : BlockQ8_0::from_float -- 32 elements; d = amax / 127; q = round(x * (1 / d)); the dot uses f16(d)
// (round = half away from zero, Rust's f32::round).  RMSNorm is applied BEFORE quantising, as the reference does
// (rms_norm -> linear), so the epilogues have nothing left to scale.
constexpr int XQ_THREADS = 1024;
__host__ __device__ inline size_t xq_seq_bytes(int K) { return (size_t)K + (size_t)(K / 32) * 8 + (size_t)(K / 16) * 4; }

// A warp's 256-element super-block g of the row: the lane's eight codes; returns their scale.  norm_w: nullable.
__device__ __forceinline__ float xq_block(int mode, const float* xrow, const float* norm_w, float rstd, int g, int lane, int (&q)[8]) {
    const int e = g * 256 + lane * 8;
    float v[8];
    {
        const float4 a0 = *reinterpret_cast<const float4*>(xrow + e), a1 = *reinterpret_cast<const float4*>(xrow + e + 4);
        v[0] = a0.x; v[1] = a0.y; v[2] = a0.z; v[3] = a0.w; v[4] = a1.x; v[5] = a1.y; v[6] = a1.z; v[7] = a1.w;
    }
    if (norm_w) {
        const float4 w0 = *reinterpret_cast<const float4*>(norm_w + e), w1 = *reinterpret_cast<const float4*>(norm_w + e + 4);
        const float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = (v[j] * rstd) * wv[j];
    }
    float am = 0.f, mx = 0.f;
    int ai = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if (fabsf(v[j]) > am) { am = fabsf(v[j]); mx = v[j]; ai = j; }       // strict: the first occurrence wins
    if (mode == XQ_Q8_K) {
        int idx = lane * 8 + ai;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float oa = __shfl_xor_sync(0xffffffffu, am, o), om = __shfl_xor_sync(0xffffffffu, mx, o);
            const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
            if (oa > am || (oa == am && oi < idx)) { am = oa; mx = om; idx = oi; }
        }
        if (am > 0.f) {
            const float iscale = -128.f / mx;
#pragma unroll
            for (int j = 0; j < 8; ++j) q[j] = (int)fminf(roundf(iscale * v[j]), 127.f);
            return 1.f / iscale;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) q[j] = 0;
        return 0.f;
    }
    am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 1));
    am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 2));
    const float df = am / 127.f;
    const float id = df != 0.f ? 1.f / df : 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) q[j] = (int)roundf(v[j] * id);
    return __half2float(__float2half_rn(df));
}

// ... of the row into the image the GEMV reads: codes (xq_swz), {d, d * sum} per 32, sums per 16
__device__ __forceinline__ void xq_image(int mode, const float* xrow, const float* norm_w, float rstd, int K, int g, int lane, unsigned char* xq) {
    float2* dsp = reinterpret_cast<float2*>(xq + K);
    int* isp = reinterpret_cast<int*>(xq + K + (K / 32) * 8);
    const int e = g * 256 + lane * 8;
    int q[8];
    const float d = xq_block(mode, xrow, norm_w, rstd, g, lane, q);
    const uint32_t p0 = (uint32_t)(q[0] & 0xff) | ((uint32_t)(q[1] & 0xff) << 8) | ((uint32_t)(q[2] & 0xff) << 16) | ((uint32_t)(q[3] & 0xff) << 24);
    const uint32_t p1 = (uint32_t)(q[4] & 0xff) | ((uint32_t)(q[5] & 0xff) << 8) | ((uint32_t)(q[6] & 0xff) << 16) | ((uint32_t)(q[7] & 0xff) << 24);
    *reinterpret_cast<uint2*>(xq + xq_swz(e)) = make_uint2(p0, p1);
    const int s8 = q[0] + q[1] + q[2] + q[3] + q[4] + q[5] + q[6] + q[7];
    const int s16 = s8 + __shfl_xor_sync(0xffffffffu, s8, 1);
    const int s32 = s16 + __shfl_xor_sync(0xffffffffu, s16, 2);
    if ((lane & 1) == 0) isp[e >> 4] = s16;
    if ((lane & 3) == 0) dsp[e >> 5] = make_float2(d, d * (float)s32);
}
// Sum of squares of a row, in ONE order whatever the launch: thread t of XQ_THREADS adds its pieces of four, a warp its lanes, 32 warps' sums last.  The scale of a row
// decides which of two codes a value on their border takes, and a flipped code moves an output by 1 / 128 of its block: another order (the warps a GEMV happens to
// have) gave a row other codes alone than in a group or a prompt.  Threads with 4 t >= K have nothing to add.
__device__ __forceinline__ void xq_square(float& ssq, const float4& v) { ssq += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w; }
__device__ __forceinline__ float xq_ssq(const float* xrow, int K, int t) {
    float ssq = 0.f;
    for (int i = t * 4; i < K; i += XQ_THREADS * 4) xq_square(ssq, *reinterpret_cast<const float4*>(xrow + i));
    return ssq;
}
__device__ __forceinline__ float xq_rstd_of(float total, int K, float eps) { return rsqrtf(total / (float)K + eps); }
__device__ __forceinline__ float xq_rstd(const float* xrow, int K, float eps, float* red) { return xq_rstd_of(block_sum(xq_ssq(xrow, K, threadIdx.x), red), K, eps); }

// One CTA per sequence: the image, written once to global for the GEMV's CTAs to fetch with one bulk copy each.
__global__ void __launch_bounds__(XQ_THREADS, 1)
xquant_kernel(const float* __restrict__ x, int ldx, int K, const float* __restrict__ norm_w, float eps, int mode, unsigned char* __restrict__ out) {
    __shared__ float red[32];
    pdl_wait();
    pdl_launch_dependents();
    const float* xrow = x + (size_t)blockIdx.x * ldx;
    const float rstd = norm_w ? xq_rstd(xrow, K, eps, red) : 1.f;
    for (int g = threadIdx.x >> 5; g < K / 256; g += XQ_THREADS / 32) xq_image(mode, xrow, norm_w, rstd, K, g, threadIdx.x & 31, out + blockIdx.x * xq_seq_bytes(K));
}
size_t xquant_bytes(int B, int K) { return (size_t)B * xq_seq_bytes(K); }
int xquant_launch(cudaStream_t st, int B, const float* x, int ldx, int K, const float* norm_w, float eps, int mode, unsigned char* out, bool pdl) {
    if ((K % 256) != 0 || B < 1 || B > 4 || (ldx % 4) != 0) return -1000;
    return launch_k(xquant_kernel, dim3(B), dim3(XQ_THREADS), 0, st, pdl, x, ldx, K, norm_w, eps, mode, out);
}

// One CTA per row: the codes as f16 rows for the tensor cores (quant.cuh, QRows).
__global__ void __launch_bounds__(XQ_THREADS, 1)
xquant_rows_kernel(const float* __restrict__ x, int ldx, int K, const float* __restrict__ norm_w, float eps, int mode, QRows rows) {
    __shared__ float red[32];
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_wait();
    pdl_launch_dependents();
    const float* xrow = x + (size_t)b * ldx;
    const float rstd = norm_w ? xq_rstd(xrow, K, eps, red) : 1.f;
    for (int g = warp; g < K / 256; g += XQ_THREADS / 32) {
        const int e = g * 256 + lane * 8;
        int q[8];
        const float d = xq_block(mode, xrow, norm_w, rstd, g, lane, q);
        auto pair = [&](int i, int j) { return (uint32_t)__half_as_ushort(__int2half_rn(q[i])) | ((uint32_t)__half_as_ushort(__int2half_rn(q[j])) << 16); };
        *reinterpret_cast<uint4*>(rows.codes + (size_t)b * K + e) = make_uint4(pair(0, 2), pair(1, 3), pair(4, 6), pair(5, 7));
        int s32 = q[0] + q[1] + q[2] + q[3] + q[4] + q[5] + q[6] + q[7];
        s32 += __shfl_xor_sync(0xffffffffu, s32, 1);
        s32 += __shfl_xor_sync(0xffffffffu, s32, 2);
        if (mode == XQ_Q8_K) {
            if (lane == 0) rows.dx[(size_t)g * rows.ldd + b] = d;
            if ((lane & 3) == 0) {
                unsigned short* bs = rows.bsum + (size_t)b * (K / 16) + g * 16 + (lane >> 2);
                bs[0] = __half_as_ushort(__int2half_rn(s32 & 63));
                bs[8] = __half_as_ushort(__int2half_rn(s32 >> 6));
            }
        } else if ((lane & 3) == 0) {
            rows.dx[(size_t)(e >> 5) * rows.ldd + b] = d;
        }
    }
}

// the scales' rows are read 128 columns at a time whatever the number of rows
static size_t qrows_pad(int rows) { return (size_t)(rows + 127) / 128 * 128; }
size_t qrows_bytes(int rows, int K) { return qrows_pad(rows) * ((size_t)K * 2 + (size_t)(K / 16) * 2 + (size_t)(K / 32) * 4); }
QRows qrows_at(unsigned char* buf, int rows, int K) {
    const size_t r = qrows_pad(rows);
    QRows q;
    q.codes = reinterpret_cast<unsigned short*>(buf);
    q.bsum = reinterpret_cast<unsigned short*>(buf + r * K * 2);
    q.dx = reinterpret_cast<float*>(buf + r * ((size_t)K * 2 + (size_t)(K / 16) * 2));
    q.ldd = (int)r;
    return q;
}
int xquant_rows_launch(cudaStream_t st, int M, const float* x, int ldx, int K, const float* norm_w, float eps, int mode, const QRows& out, bool pdl) {
    if ((K % 256) != 0 || M < 1 || M > out.ldd || (ldx % 4) != 0) return -1000;
    return launch_k(xquant_rows_kernel, dim3(M), dim3(XQ_THREADS), 0, st, pdl, x, ldx, K, norm_w, eps, mode, out);
}

#ifndef QG_R_DEF                    // tools/qgemv_bench.cu sweeps these
#define QG_R_DEF 4
#define QG_DEPTH_DEF 2
#define QG_W1_DEF 16
#define QG_W4_DEF 12
#endif
constexpr int QG_R = QG_R_DEF;     // rows per tile
constexpr int QG_KT = 8;           // super-blocks per tile row (32 lanes x 64 elements)
constexpr int QG_DEPTH = QG_DEPTH_DEF;   // tiles in flight per warp
__host__ __device__ constexpr int qg_warps(int B) { return B >= 4 ? QG_W4_DEF : QG_W1_DEF; }

// One CTA per SM owns a contiguous block of output rows.  Work unit = tile of QG_R rows x QG_KT super-blocks; a warp takes
// a contiguous range of tiles (k fastest), streams each through its private cp.async ring, keeps its activation slice in
// registers and one f32 accumulator per (row, sequence), and flushes them to the CTA's shared row accumulators when it
// moves on to another row group.  The flush is an atomic add: two warps' shares of a row give the same sum in either order; three or more, which short
// row blocks of more than 4096 columns can have (512 x 6144), may differ in the last bit from run to run.
// MORE: q, k and v share the launch (QMore)
template <int B, int QT, bool MORE>
__global__ void __launch_bounds__(qg_warps(B) * 32, 1)
qgemv_kernel(QGemvArgs qa) {
    using TR = QTraits<QT>;
    constexpr int QG_MAXW = qg_warps(B);
    const int QG_WARPS = (int)(blockDim.x >> 5);       // chosen at launch so rings + activations fit in shared memory
    const int QG_THREADS = (int)blockDim.x;
    constexpr int ROWB = QG_KT * TR::SB;               // bytes of one tile row
    constexpr int SLOT = QG_R * ROWB;                  // bytes per ring slot
    const GemvArgs& a = qa.g;
    extern __shared__ __align__(1024) unsigned char qsm[];
    // layout: [rings: QG_WARPS * DEPTH * SLOT][per b: xq K | {d, d*sum} K/32 float2 | isum16 K/16 i32][acc B * rpc f32]
    const int K = a.K;
    const size_t xb = (size_t)K + (size_t)(K / 32) * 8 + (size_t)(K / 16) * 4;       // bytes of quantised activation per sequence
    unsigned char* xbase = qsm + (size_t)QG_WARPS * QG_DEPTH * SLOT;
    const int rows_per_unit = (qa.epi == GEMV_SILU_MUL) ? 2 : 1;
    const int mats = !MORE ? 1 : qa.more.n[1] ? 3 : 2;
    float* acc_s = reinterpret_cast<float*>(xbase + (size_t)B * xb);
    __shared__ uint64_t xbar;
    __shared__ float red[32];
    __shared__ float wbest_v[QG_MAXW][B];
    __shared__ int wbest_i[QG_MAXW][B];
    __shared__ int is_last_s;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t spr = (uint32_t)(K >> 8);                                          // super-blocks per row
    const uint32_t nkt = (spr + QG_KT - 1) / QG_KT;                                   // k-tiles per row
    const size_t row_bytes = (size_t)spr * TR::SB;
    // The matrix at hand and this CTA's rows of it.  Every matrix is dealt out as in a launch of its own, so that its rows' sums are formed in the same order, and
    // the codes of the next linear are the same, whether q, k and v share a launch or not.
    struct Mat { const unsigned char* w; int rpc, r0, nrows, out, acc0; };             // (out, acc0: what the matrices ahead take of y and of the sums)
    auto mat = [&](int k) {
        Mat m{reinterpret_cast<const unsigned char*>(a.W), qa.rpc[0], 0, a.N, 0, 0};
        if (MORE && k >= 1) m = Mat{qa.more.w[0], qa.rpc[1], 0, qa.more.n[0], a.N, B * qa.rpc[0]};
        if (MORE && k >= 2) m = Mat{qa.more.w[1], qa.rpc[2], 0, qa.more.n[1], a.N + qa.more.n[0], B * (qa.rpc[0] + qa.rpc[1])};
        m.r0 = (int)blockIdx.x * m.rpc;
        m.nrows = max(0, min(m.nrows, m.r0 + m.rpc) - m.r0);
        return m;
    };
    // this warp's tiles [t, end) of it, of R rows; `turn`: the warp that takes the first ones, as short matrices leave warps without any.
    struct Deal { uint32_t R, t, end; };
    uint32_t turn = 0;
    auto deal = [&](int nrows) {
        Deal d{QG_R};
        // rows per tile: QG_R when that leaves every warp at least two tiles, fewer for short row blocks (q/k/v/o projections)
        while (d.R > 1 && (((uint32_t)nrows + d.R - 1) / d.R) * nkt < 2u * (uint32_t)QG_WARPS) d.R >>= 1;
        const uint32_t ntile = ((uint32_t)nrows + d.R - 1) / d.R * nkt, tpw = (ntile + QG_WARPS - 1) / QG_WARPS;
        const uint32_t u = (uint32_t)warp >= turn ? warp - turn : warp + QG_WARPS - turn;
        d.t = min(ntile, u * tpw);
        d.end = min(ntile, (u + 1) * tpw);
        if (MORE) {
            turn += ntile ? (ntile + tpw - 1) / tpw : 0u;
            if (turn >= (uint32_t)QG_WARPS) turn -= QG_WARPS;
        }
        return d;
    };
    const Deal d0 = deal(mat(0).nrows);
    Deal d1 = d0, d2 = d0;
    auto dealt = [&](int k) { return !MORE || k == 0 ? d0 : k == 1 ? d1 : d2; };
    unsigned char* ring = qsm + (size_t)warp * QG_DEPTH * SLOT;
    const uint32_t ring_u32 = smem_u32(ring);

    Mat mi = mat(0);                                    // the tiles requested so far
    Deal di = d0;
    int ki = 0;
    uint32_t islot = 0;
    auto issue = [&]() {
        while (di.t == di.end && ki + 1 < mats) { ++ki; mi = mat(ki); di = dealt(ki); }
        if (di.t < di.end) {
            const uint32_t rg = di.t / nkt, kt = di.t - rg * nkt;
            const uint32_t nr = min(di.R, (uint32_t)mi.nrows - rg * di.R);
            const uint32_t cpr = min((uint32_t)QG_KT, spr - kt * QG_KT) * (TR::SB / 16);      // 16-byte chunks per tile row
            const uint32_t dst = ring_u32 + islot * SLOT;
            const unsigned char* src = mi.w + (size_t)(mi.r0 + rg * di.R) * row_bytes + (size_t)kt * QG_KT * TR::SB;
            for (uint32_t r = 0; r < nr; ++r, src += row_bytes)
                for (uint32_t c = lane; c < cpr; c += 32)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + r * ROWB + c * 16), "l"(src + (size_t)c * 16) : "memory");
            ++di.t;
        }
        islot = islot + 1 == QG_DEPTH ? 0 : islot + 1;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int primed = 0;
    if (MORE) {                                         // (the first requests leave ahead of the other matrices' divisions)
        for (; primed < QG_DEPTH && di.t < di.end; ++primed) issue();
        d1 = deal(mat(1).nrows);
        if (mats > 2) d2 = deal(mat(2).nrows);
    }
    for (; primed < QG_DEPTH; ++primed) issue();
    for (int i = tid; i < B * (qa.rpc[0] + (mats > 1 ? qa.rpc[1] : 0) + (mats > 2 ? qa.rpc[2] : 0)); i += QG_THREADS) acc_s[i] = 0.f;
    if (tid == 0) { mbar_init(&xbar, 1); fence_barrier_init(); }
    __syncthreads();

    pdl_wait();
    pdl_launch_dependents();

    const int r0 = mat(0).r0, nrows = mat(0).nrows, rpc = qa.rpc[0];
    float old[B];                                       // (beside the activations, not behind the dots)
    if (qa.epi == GEMV_RESID)
#pragma unroll
        for (int b = 0; b < B; ++b) old[b] = tid < nrows ? a.y[(size_t)b * a.ldy + r0 + tid] : 0.f;
    // ---- the quantised activations: one bulk copy of the ready-made image, or every CTA for itself (xquant_apart) ----
    constexpr bool INSIDE = B == 1 && QT == QT_Q8_0;
    if (!INSIDE || qa.xq) {
        if (tid == 0) {
            mbar_arrive_expect_tx(&xbar, (uint32_t)(B * xb));
            bulk_load(xbase, qa.xq, (uint32_t)(B * xb), &xbar);
        }
        mbar_wait(&xbar, 0);
    } else if constexpr (INSIDE) {
        const int nvw = min(32, (K + 127) / 128);           // of xq_ssq's 32 warps, those with anything to add
        if (a.norm_w) {
#pragma unroll 1
            for (int vw = warp; vw < nvw; vw += 4 * QG_WARPS) {      // four of them at once, of one or two pieces each (xquant_apart): all loads are in flight together
                float4 v[4][2];
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int w = vw + j * QG_WARPS, i = (w * 32 + lane + h * XQ_THREADS) * 4;
                        v[j][h] = w < nvw && i < K ? *reinterpret_cast<const float4*>(a.x + i) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float ssq = 0.f;
                    xq_square(ssq, v[j][0]);
                    xq_square(ssq, v[j][1]);            // (what is not there adds nothing)
                    ssq = warp_sum(ssq);
                    if (lane == 0 && vw + j * QG_WARPS < nvw) red[vw + j * QG_WARPS] = ssq;
                }
            }
            __syncthreads();
        }
#pragma unroll 1
        for (int g = warp; g < (int)spr; g += QG_WARPS) {
            const float rstd = a.norm_w ? xq_rstd_of(warp_sum(lane < nvw ? red[lane] : 0.f), K, a.eps) : 1.f;
            xq_image(xq_mode_for(QT), a.x, a.norm_w, rstd, K, g, lane, xbase);
        }
        __syncthreads();
    }

    // ---- stream this warp's tiles ----
    {
        const int sbk = lane >> 2, qq = lane & 3;              // this lane's super-block within the tile row and its quarter
        XSlice<QT, B> xs;
        float acc[QG_R * B];
#pragma unroll
        for (int i = 0; i < QG_R * B; ++i) acc[i] = 0.f;
        uint32_t cur_kt = 0xffffffffu, slot = 0;
        for (int k = 0; k < mats; ++k) {
            const Mat m = mat(k);
            const Deal d = dealt(k);
            uint32_t cur_rg = 0xffffffffu;
            auto flush = [&]() {
                int idx;
                warp_reduce_scatter<QG_R * B>(acc, lane, idx);
                const int r = idx / B, b = idx % B;
                const uint32_t row = cur_rg * d.R + r;
                if ((lane & (32 / (QG_R * B) - 1)) == 0 && (uint32_t)r < d.R && row < (uint32_t)m.nrows) atomicAdd(&acc_s[m.acc0 + (size_t)b * m.rpc + row], acc[0]);
#pragma unroll
                for (int i = 0; i < QG_R * B; ++i) acc[i] = 0.f;
            };
            for (uint32_t t = d.t; t < d.end; ++t) {
                asm volatile("cp.async.wait_group %0;" ::"n"(QG_DEPTH - 1) : "memory");
                __syncwarp();
                const uint32_t rg = t / nkt, kt = t - rg * nkt;
                if (rg != cur_rg) {
                    if (cur_rg != 0xffffffffu) flush();
                    cur_rg = rg;
                }
                const bool active = kt * QG_KT + sbk < spr;
                if (kt != cur_kt) {
                    if (active) xs.load(xbase, xb, K, (int)(kt * QG_KT) + sbk, qq);
                    cur_kt = kt;
                }
                const uint32_t nr = min(d.R, (uint32_t)m.nrows - rg * d.R);
                const unsigned char* sb = ring + slot * SLOT + sbk * TR::SB;
                if (active) {
#pragma unroll
                    for (int r = 0; r < QG_R; ++r)
                        if ((uint32_t)r < nr) sb_quarter_dot<QT, B>(sb + r * ROWB, qq, xs, acc + r * B);
                }
                __syncwarp();
                issue();
                slot = slot + 1 == QG_DEPTH ? 0 : slot + 1;
            }
            if (cur_rg != 0xffffffffu) flush();
        }
    }
    __syncthreads();

    // ---- epilogue (same contracts as the bf16 GEMV) ----
    for (int k = 1; k < mats; ++k) {
        const Mat m = mat(k);
        for (int i = tid; i < m.nrows; i += QG_THREADS)
#pragma unroll
            for (int b = 0; b < B; ++b) a.y[(size_t)b * a.ldy + m.out + m.r0 + i] = acc_s[m.acc0 + b * m.rpc + i];
    }
    float bestv[B];
    int besti[B];
#pragma unroll
    for (int b = 0; b < B; ++b) { bestv[b] = -INFINITY; besti[b] = 0x7fffffff; }
    if (qa.epi == GEMV_SILU_MUL) {
        for (int u = tid; u < nrows / 2; u += QG_THREADS)
#pragma unroll
            for (int b = 0; b < B; ++b) a.y[(size_t)b * a.ldy + (r0 / 2 + u)] = silu_f(acc_s[(size_t)b * rpc + 2 * u]) * acc_s[(size_t)b * rpc + 2 * u + 1];
    } else {
        for (int i = tid; i < nrows; i += QG_THREADS)
#pragma unroll
            for (int b = 0; b < B; ++b) {
                const float v = acc_s[(size_t)b * rpc + i];
                float* yp = a.y + (size_t)b * a.ldy + r0 + i;
                if (qa.epi == GEMV_RESID) *yp = (i == tid ? old[b] : *yp) + v; else *yp = v;
                if (qa.epi == GEMV_LOGITS_ARGMAX && v > bestv[b]) { bestv[b] = v; besti[b] = r0 + i; }
            }
    }
    if (qa.epi == GEMV_LOGITS_ARGMAX) {
#pragma unroll
        for (int b = 0; b < B; ++b)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, bestv[b], o);
                const int oi = __shfl_xor_sync(0xffffffffu, besti[b], o);
                if (ov > bestv[b] || (ov == bestv[b] && oi < besti[b])) { bestv[b] = ov; besti[b] = oi; }
            }
        if (lane == 0)
#pragma unroll
            for (int b = 0; b < B; ++b) { wbest_v[warp][b] = bestv[b]; wbest_i[warp][b] = besti[b]; }
        __syncthreads();
        if (tid < B) {
            float bv = -INFINITY; int bi = 0x7fffffff;
            for (int w = 0; w < QG_WARPS; ++w) {
                const float v = wbest_v[w][tid]; const int i = wbest_i[w][tid];
                if (v > bv || (v == bv && i < bi)) { bv = v; bi = i; }
            }
            a.part_val[tid * gridDim.x + blockIdx.x] = bv;
            a.part_idx[tid * gridDim.x + blockIdx.x] = bi;
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) is_last_s = (atomicAdd(a.ticket, 1u) == gridDim.x - 1);
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
                    tok_s[b] = (uint32_t)bi;
                    SeqState* s = a.state + b;
                    if (a.out_tokens) a.out_tokens[(size_t)b * a.out_stride + s->step] = (uint32_t)bi;
                    if (a.advance) { s->token = (uint32_t)bi; s->kv_len += 1; s->pos[0] += 1; s->pos[1] += 1; s->pos[2] += 1; }
                    s->step += 1;
                }
            }
            if (tid == 0) *a.ticket = 0u;
            __syncthreads();
            if (a.advance && a.embed != nullptr)
                for (int b = 0; b < B; ++b) {
                    const bf16* rowp = a.embed + (size_t)tok_s[b] * a.H;
                    for (int i = tid; i < a.H; i += QG_THREADS) a.x_next[(size_t)b * a.H + i] = __bfloat162float(rowp[i]);
                }
        }
    }
}

template <int B, int QT>
static int qgemv_launch_t(cudaStream_t st, const QGemvArgs& args, int num_sms, bool pdl) {
    using TR = QTraits<QT>;
    QGemvArgs qa = args;
    const GemvArgs& a = qa.g;
    const int rpu = qa.epi == GEMV_SILU_MUL ? 2 : 1;
    auto rpc = [&](int n) { return (size_t)((n / rpu + num_sms - 1) / num_sms * rpu); };
    const size_t xb = (size_t)a.K + (size_t)(a.K / 32) * 8 + (size_t)(a.K / 16) * 4;
    const size_t fixed = (size_t)B * xb + 32, slot = (size_t)QG_DEPTH * QG_R * QG_KT * TR::SB, most = 226 * 1024;
    auto warps = [&](int n) {                           // what fits beside n rows' sums
        int w = qg_warps(B);
        while (w > 4 && fixed + B * rpc(n) * 4 + w * slot > most) --w;
        return w;
    };
    const int QG_WARPS = warps(a.N);
    size_t smem = fixed + B * rpc(a.N) * 4 + QG_WARPS * slot;
    if (qa.more.n[0]) {
        if (qa.epi != GEMV_STORE) return -1000;
        bool one = true;
        for (int n : qa.more.n) if (n) { one = one && warps(n) == QG_WARPS; smem += B * rpc(n) * 4; }
        if (!one || smem > most) {                      // launches of their own: the same sums
            QGemvArgs q = qa;
            q.more = QMore{};
            int e = qgemv_launch_t<B, QT>(st, q, num_sms, pdl);
            for (int i = 0; i < 2 && qa.more.n[i] && !e; ++i) {
                q.g.y += q.g.N; q.g.N = qa.more.n[i]; q.g.W = reinterpret_cast<const bf16*>(qa.more.w[i]);
                e = qgemv_launch_t<B, QT>(st, q, num_sms, pdl);
            }
            return e;
        }
    }
    const int QG_THREADS = QG_WARPS * 32;
    if (smem > most) return -1000;
    for (int i = 0; i < 3; ++i) qa.rpc[i] = (int)rpc(i ? qa.more.n[i - 1] : a.N);
    static SmemOptIn seen[2];
    auto* kern = qa.more.n[0] ? qgemv_kernel<B, QT, true> : qgemv_kernel<B, QT, false>;
    if (const int e = ensure_dyn_smem(kern, smem, seen[qa.more.n[0] != 0])) return e;
    return launch_k(kern, dim3(num_sms), dim3(QG_THREADS), smem, st, pdl, qa);
}

template <int B>
static int qgemv_launch_b(cudaStream_t st, const QGemvArgs& qa, int num_sms, bool pdl) {
    switch (qa.qtype) {
        case QT_Q4_K: return qgemv_launch_t<B, QT_Q4_K>(st, qa, num_sms, pdl);
        case QT_Q6_K: return qgemv_launch_t<B, QT_Q6_K>(st, qa, num_sms, pdl);
        case QT_Q8_0: return qgemv_launch_t<B, QT_Q8_0>(st, qa, num_sms, pdl);
        default: return -1000;
    }
}

int qgemv_launch(cudaStream_t st, int B, const QGemvArgs& qa, int num_sms, bool pdl) {
    if ((qa.g.K % 256) != 0 || qa.g.N <= 0 || (qa.g.ldx % 4) != 0) return -1000;
    if (qa.epi == GEMV_SILU_MUL && (qa.g.N % 2) != 0) return -1000;
    if (!qa.xq && xquant_apart(B, qa.g.K, qa.qtype)) return -1000;
    switch (B) {
        case 1: return qgemv_launch_b<1>(st, qa, num_sms, pdl);
        case 2: return qgemv_launch_b<2>(st, qa, num_sms, pdl);
        case 4: return qgemv_launch_b<4>(st, qa, num_sms, pdl);
        default: return -1000;
    }
}

// ------------------------------------------------------------------------------------------------ dequantise
// elements [8g, 8g + 8) of one 256-element super-block (device layout) -> f32, exactly d * sc * q - dmin * m / d * sc * (q - 32) / d * q
template <int QT>
__device__ __forceinline__ void dequant8(const unsigned char* sb, int g, float (&v)[8]) {
    if constexpr (QT == QT_Q4_K) {
        const float d = f16_bits_to_float(*reinterpret_cast<const unsigned short*>(sb));
        const float dmin = f16_bits_to_float(*reinterpret_cast<const unsigned short*>(sb + 2));
        const unsigned char* sc8 = sb + 4;
        const int j = g >> 2;                    // sub-block
        int sc, m;
        if (j < 4) { sc = sc8[j] & 63; m = sc8[j + 4] & 63; }
        else { sc = (sc8[j + 4] & 0xF) | ((sc8[j - 4] >> 6) << 4); m = (sc8[j + 4] >> 4) | ((sc8[j] >> 6) << 4); }
        const unsigned char* qs = sb + 16 + 32 * (j >> 1) + 8 * (g & 3);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int q = (j & 1) ? (qs[i] >> 4) : (qs[i] & 0xF);
            v[i] = d * (float)sc * (float)q - dmin * (float)m;
        }
    } else if constexpr (QT == QT_Q6_K) {
        const float d = f16_bits_to_float(*reinterpret_cast<const unsigned short*>(sb + 208));
        const signed char* sc = reinterpret_cast<const signed char*>(sb + 192);
        const int half = g >> 4, gi = g & 15;    // 16 groups of 8 per half
        const int quarter = gi >> 2;             // which of q1..q4 (elements +0, +32, +64, +96)
        const int l0 = (gi & 3) * 8;             // l of the first element
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int l = l0 + i;
            const unsigned char ql = sb[64 * half + l + ((quarter & 1) ? 32 : 0)];
            const unsigned char qh = sb[128 + 32 * half + l];
            const int lo = (quarter & 2) ? (ql >> 4) : (ql & 0xF);
            const int hi = (qh >> (2 * quarter)) & 3;
            const int q = (lo | (hi << 4)) - 32;
            v[i] = d * (float)sc[8 * half + 2 * quarter + l / 16] * (float)q;
        }
    } else {
        const int blk = g >> 2;
        const float d = f16_bits_to_float(*reinterpret_cast<const unsigned short*>(sb + 256 + 2 * blk));
        const signed char* q = reinterpret_cast<const signed char*>(sb + 8 * g);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = d * (float)q[i];
    }
}

// One thread per (super-block, 8-element group): a whole quantised matrix -> bf16
template <int QT>
__global__ void __launch_bounds__(256)
q_dequant_kernel(const unsigned char* __restrict__ w, size_t nsb, bf16* __restrict__ out) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t gid = (size_t)blockIdx.x * 256 + threadIdx.x;
    const size_t sbi = gid >> 5;
    const int g = (int)(gid & 31);               // elements [8g, 8g+8)
    if (sbi >= nsb) return;
    float v[8];
    dequant8<QT>(w + sbi * QTraits<QT>::SB, g, v);
    uint4 o = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
    *reinterpret_cast<uint4*>(out + sbi * 256 + 8 * g) = o;
}

int q_dequant_bf16_launch(cudaStream_t st, int qt, const unsigned char* w, size_t rows, int K, bf16* out) {
    const size_t nsb = rows * (K / 256);
    const size_t threads = nsb * 32;
    const unsigned int grid = (unsigned int)((threads + 255) / 256);
    switch (qt) {
        case QT_Q4_K: return launch_k(q_dequant_kernel<QT_Q4_K>, dim3(grid), dim3(256), 0, st, prefill_pdl(), w, nsb, out);
        case QT_Q6_K: return launch_k(q_dequant_kernel<QT_Q6_K>, dim3(grid), dim3(256), 0, st, prefill_pdl(), w, nsb, out);
        case QT_Q8_0: return launch_k(q_dequant_kernel<QT_Q8_0>, dim3(grid), dim3(256), 0, st, prefill_pdl(), w, nsb, out);
        default: return -1000;
    }
}

// Quantised embedding: the table stays in its ggml blocks and only the gathered rows are dequantised, to f32
// (`QuantizedEmbedding::forward`, crane-core/src/models/modules/embedding.rs:31-105: index_select of Q-blocks + dequantize).
// Row ids come from `ids` (prefill) or, when ids == nullptr, from state[row].token (the decode step's input).
template <int QT>
__global__ void __launch_bounds__(256)
embed_rows_q_kernel(const unsigned char* __restrict__ table, int H, const uint32_t* __restrict__ ids, const SeqState* __restrict__ state,
                    float* __restrict__ x) {
    pdl_wait();
    pdl_launch_dependents();
    const int r = blockIdx.x;
    const uint32_t tok = ids ? ids[r] : state[r].token;
    const unsigned char* row = table + (size_t)tok * (H / 256) * QTraits<QT>::SB;
    for (int it = threadIdx.x; it < H / 8; it += 256) {
        float v[8];
        dequant8<QT>(row + (size_t)(it >> 5) * QTraits<QT>::SB, it & 31, v);
        float4* o = reinterpret_cast<float4*>(x + (size_t)r * H + it * 8);
        o[0] = make_float4(v[0], v[1], v[2], v[3]);
        o[1] = make_float4(v[4], v[5], v[6], v[7]);
    }
}

int embed_rows_q_launch(cudaStream_t st, int qt, const unsigned char* table, int H, const uint32_t* ids, const SeqState* state, int rows,
                        float* x, bool pdl) {
    if (rows <= 0 || (H % 256) != 0) return -1000;
    switch (qt) {
        case QT_Q4_K: return launch_k(embed_rows_q_kernel<QT_Q4_K>, dim3(rows), dim3(256), 0, st, pdl, table, H, ids, state, x);
        case QT_Q6_K: return launch_k(embed_rows_q_kernel<QT_Q6_K>, dim3(rows), dim3(256), 0, st, pdl, table, H, ids, state, x);
        case QT_Q8_0: return launch_k(embed_rows_q_kernel<QT_Q8_0>, dim3(rows), dim3(256), 0, st, pdl, table, H, ids, state, x);
        default: return -1000;
    }
}

}  // namespace cb
