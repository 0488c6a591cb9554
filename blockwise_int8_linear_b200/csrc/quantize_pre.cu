// Row-wise block quantizers with the elementwise step that produces their input fused in front.
//
// In a transformer layer the input of every quantized projection comes out of a short elementwise step: the
// normalisation in front of q/k/v and gate/up, the gated activation in front of the down projection.  Run as separate
// kernels these write a [M, K] tensor in the activation type that the quantizer (triton_functions.py:411-423 in the
// reference, one program per row) reads back at once.  The kernels here compute that tensor in registers, round every
// value to the activation type exactly as the separate kernel would have stored it, and quantize it with the same
// arithmetic as the stand-alone quantizer (quant_math.cuh), so that the int8 values and scales are those of
// quantize_block_rowwise applied to the rounded tensor.
//
//   BI8_PRE_RMSNORM   y = cast(x * rsqrt(sum(x^2) / K + eps) [* weight])        one rounding, fp32 arithmetic
//   BI8_PRE_SILU_MUL  y = cast(cast(x / (1 + exp(-x))) * x2)                    two roundings: silu(x), then the product
//
// Both release their programmatic dependents at once (the decode GEMM launched behind them sets up and streams its first
// weights while they run; it waits for their completion before it reads the activations).  For decode-sized batches they
// are themselves launched as programmatic dependents of whatever precedes them in the stream, wait for it first thing,
// and release their own dependents only then: behind one of this library's reduction kernels (the previous layer's)
// they are resident before that kernel has finished.
#include "bi8_common.cuh"
#include "quant_math.cuh"
#include "tc_common.cuh"

#include <cstring>

namespace bi8 {
namespace {

constexpr int kPreThreads = 256;
constexpr int kPreHold = 4;        // 8-element units of a row a thread keeps in registers between the two passes

// eight consecutive elements of a row, beginning at element `k` of `K`; elements from K on read as zero
__device__ __forceinline__ void load8(float* f, const void* base, int64_t row_off, int k, int K, int dt, bool vec) {
    const int esz = dt == BI8_F32 ? 4 : 2;
    const unsigned char* src = static_cast<const unsigned char*>(base) + (row_off + k) * esz;
    if (vec && k + 8 <= K) {
        const uint4 a = ld_nc_v4(src);
        if (dt == BI8_F32) {
            const uint4 b = ld_nc_v4(src + 16);
            f[0] = __uint_as_float(a.x); f[1] = __uint_as_float(a.y); f[2] = __uint_as_float(a.z); f[3] = __uint_as_float(a.w);
            f[4] = __uint_as_float(b.x); f[5] = __uint_as_float(b.y); f[6] = __uint_as_float(b.z); f[7] = __uint_as_float(b.w);
        } else {
            const uint32_t w4[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                if (dt == BI8_BF16) {
                    f[2 * h] = bf16lo(w4[h]);
                    f[2 * h + 1] = bf16hi(w4[h]);
                } else {
                    const float2 t2 = __half22float2(*reinterpret_cast<const __half2*>(&w4[h]));
                    f[2 * h] = t2.x;
                    f[2 * h + 1] = t2.y;
                }
            }
        }
        return;
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        float v = 0.0f;
        if (k + e < K) {
            if (dt == BI8_F32) v = reinterpret_cast<const float*>(src)[e];
            else if (dt == BI8_BF16) v = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(src)[e]);
            else v = __half2float(reinterpret_cast<const __half*>(src)[e]);
        }
        f[e] = v;
    }
}

// the same eight elements of a 16-bit type as four packed words (what a thread keeps between the two passes of a row)
__device__ __forceinline__ void load_raw8(uint32_t* w, const void* base, int64_t row_off, int k, int K, bool vec) {
    const unsigned char* src = static_cast<const unsigned char*>(base) + (row_off + k) * 2;
    if (vec && k + 8 <= K) {
        const uint4 a = ld_nc_v4(src);
        w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
        return;
    }
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        const uint32_t lo = k + 2 * h < K ? reinterpret_cast<const unsigned short*>(src)[2 * h] : 0u;
        const uint32_t hi = k + 2 * h + 1 < K ? reinterpret_cast<const unsigned short*>(src)[2 * h + 1] : 0u;
        w[h] = lo | (hi << 16);
    }
}

__device__ __forceinline__ void unpack8(float* f, const uint32_t* w, int dt) {
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        if (dt == BI8_BF16) {
            f[2 * h] = bf16lo(w[h]);
            f[2 * h + 1] = bf16hi(w[h]);
        } else {
            const float2 t2 = __half22float2(*reinterpret_cast<const __half2*>(&w[h]));
            f[2 * h] = t2.x;
            f[2 * h + 1] = t2.y;
        }
    }
}

// Quantizes the eight values of a unit whose block's other units sit in the neighbouring lanes (LPB lanes per block)
// and stores them; all 32 lanes of the warp must call it.
template <int QB>
__device__ __forceinline__ void quantize_unit(const float (&y)[8], bool valid, bool short_mantissa, int8_t* q, int64_t ldq, float* sx, int m, int k,
                                              int M, int K, bool vec) {
    constexpr int LPB = QB / 8;
    float amax = 0.0f;
#pragma unroll
    for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(y[e]));
#pragma unroll
    for (int off = 1; off < LPB; off <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    BlockQ bq;
    bq.set(amax, short_mantissa);
    if (!valid) return;
    uint32_t lo, hi;
    quantize8(y, bq, lo, hi);
    int8_t* dst = q + (int64_t)m * ldq + k;
    if (vec) {                               // the row pitch covers the eight bytes of a row's last unit
        *reinterpret_cast<uint2*>(dst) = make_uint2(lo, hi);
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (k + e < K) dst[e] = (int8_t)(((e < 4 ? lo : hi) >> (8 * (e & 3))) & 0xffu);
    }
    if (((k / 8) % LPB) == 0) sx[(int64_t)(k / QB) * M + m] = amax;
}

// One CTA per row.  Pass 1: the row's sum of squares (a thread's units in ascending order, lanes by butterfly, warps in
// ascending order: the same bits on every launch with the same THREADS, which the launcher picks from M and K).  Pass 2: normalise, round, quantize.  Rows of up
// to kPreHold * THREADS * 8 elements stay in registers between the passes; longer rows are read again.  THREADS = 128
// for rows of up to 4096 elements: a row is in flight for a load latency plus a reduction, so what bounds a large
// batch is the number of rows resident per SM (ten CTAs of 128 threads against five of 256).
//
// EARLY: the weight is requested with the row, not behind the reduction, for 56 registers instead of 46 and four resident CTAs instead
// of five.  Back to back, bf16, block 64, without / with: 8 x 4096 2.7 / 2.45 us, 256 x 4096 3.5 / 3.15, 512 x 4096 5.1 / 4.4, 760 x 4096
// 6.8 / 6.45, 1024 x 4096 7.65 / 7.35, 2048 x 8192 21.2 / 20.0, 2048 x 5120 15.2 / 15.2 (cold, in a decode layer of 8 sequences, 69.7 /
// 68.6 a layer).  Not where five CTAs per SM take all rows at once and four do not (600 to 740 x 4096: 5.3-5.5 / 5.7-6.3), and
// not for rows that do not stay in registers, which have no use for it (2048 x 11008: 39.0 / 45.7, 2048 x 16384: 53.8 / 64.0).
template <int QB, int THREADS, int DT, bool EARLY>
__global__ void __launch_bounds__(THREADS, THREADS == 128 ? 10 : 4) rmsnorm_quantize_kernel(const void* __restrict__ x, int64_t ldx,
                                                                       const void* __restrict__ weight, float eps,
                                                                       int8_t* __restrict__ q, int64_t ldq, float* __restrict__ sx, int M, int K,
                                                                       int nb, int vec_in, int vec_out) {
    after_predecessor();
    constexpr int LPB = QB / 8;
    constexpr int dt = DT;                                        // the element type is a template parameter: no per-element tests
    __shared__ float warp_sum[THREADS / 32];
    const int m = blockIdx.x, tid = threadIdx.x;
    const int upr = nb * LPB;                                   // units per row, padded to whole blocks
    // 16-bit rows that fit are kept as packed words (four registers per unit); fp32 rows and longer ones are read again
    const bool hold = dt != BI8_F32 && upr <= kPreHold * THREADS;
    const int64_t row_off = (int64_t)m * ldx;
    uint32_t raw[kPreHold][4];
    uint32_t wraw[EARLY ? kPreHold : 1][4];
    float ss = 0.0f;
    if (hold) {
#pragma unroll
        for (int i = 0; i < kPreHold; ++i) {
            const int k = (i * THREADS + tid) * 8;
            if (k < K) load_raw8(raw[i], x, row_off, k, K, vec_in != 0);
            else raw[i][0] = raw[i][1] = raw[i][2] = raw[i][3] = 0u;
        }
        if constexpr (EARLY) {
#pragma unroll
            for (int i = 0; i < kPreHold; ++i) {
                const int k = (i * THREADS + tid) * 8;
                if (weight != nullptr && k < K) load_raw8(wraw[i], weight, 0, k, K, vec_in != 0);
                else wraw[i][0] = wraw[i][1] = wraw[i][2] = wraw[i][3] = 0u;
            }
        }
#pragma unroll
        for (int i = 0; i < kPreHold; ++i) {
            float t[8];
            unpack8(t, raw[i], dt);
#pragma unroll
            for (int e = 0; e < 8; ++e) ss = __fmaf_rn(t[e], t[e], ss);
        }
    } else {
        for (int u = tid; u < upr; u += THREADS) {
            const int k = u * 8;
            if (k >= K) break;
            float t[8];
            load8(t, x, row_off, k, K, dt, vec_in != 0);
#pragma unroll
            for (int e = 0; e < 8; ++e) ss = __fmaf_rn(t[e], t[e], ss);
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    if ((tid & 31) == 0) warp_sum[tid >> 5] = ss;
    __syncthreads();
    float total = 0.0f;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) total += warp_sum[w];
    const float rstd = rsqrtf(__fadd_rn(__fdiv_rn(total, (float)K), eps));
    const bool short_mantissa = dt != BI8_F32;
    // normalises, rounds and quantizes the unit whose elements are in y (all lanes of a warp call it together)
    auto finish_unit = [&](float (&y)[8], int k, bool valid, const uint32_t* early) {
        if (valid) {
            float w8[8];
            if (early) unpack8(w8, early, dt);
            else if (weight) load8(w8, weight, 0, k, K, dt, vec_in != 0);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                float v = __fmul_rn(y[e], rstd);
                if (weight) v = __fmul_rn(v, w8[e]);
                y[e] = round_to(v, dt);
            }
        }
        quantize_unit<QB>(y, valid, short_mantissa, q, ldq, sx, m, k, M, K, vec_out != 0);
    };
    if (hold) {
#pragma unroll
        for (int i = 0; i < kPreHold; ++i) {
            if (i * THREADS < upr) {                            // the same for all threads of the CTA
                const int u = i * THREADS + tid, k = u * 8;
                float y[8];
                unpack8(y, raw[i], dt);
                finish_unit(y, k, u < upr && k < K, EARLY ? wraw[EARLY ? i : 0] : nullptr);
            }
        }
    } else {
        for (int i = 0; i * THREADS < upr; ++i) {
            const int u = i * THREADS + tid, k = u * 8;
            const bool valid = u < upr && k < K;
            float y[8];
            if (valid) {
                load8(y, x, row_off, k, K, dt, vec_in != 0);
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) y[e] = 0.0f;
            }
            finish_unit(y, k, valid, nullptr);
        }
    }
}

// One thread per unit of eight elements, as in the decode quantizer: few rows, fp32, operands off 16-byte boundaries.
template <int QB, int DT>
__global__ void __launch_bounds__(kPreThreads) silu_mul_quantize_kernel(const void* __restrict__ gate, const void* __restrict__ up,
                                                                        int64_t ldx, int8_t* __restrict__ q, int64_t ldq,
                                                                        float* __restrict__ sx, int M, int K, FastDiv upr, int vec_in,
                                                                        int vec_out) {
    after_predecessor();
    constexpr int dt = DT;
    const int64_t u = (int64_t)blockIdx.x * kPreThreads + threadIdx.x;
    const int m = u < (1ll << 31) ? (int)upr.div((unsigned)u) : (int)(u / upr.d), k = (int)(u - (int64_t)m * upr.d) * 8;
    const bool valid = m < M && k < K;
    float y[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) y[e] = 0.0f;
    if (valid) {
        float v[8];
        load8(y, gate, (int64_t)m * ldx, k, K, dt, vec_in != 0);
        load8(v, up, (int64_t)m * ldx, k, K, dt, vec_in != 0);
        silu_mul8(y, v, dt);
    }
    quantize_unit<QB>(y, valid, dt != BI8_F32, q, ldq, sx, m, k, M, K, vec_out != 0);
}

// The same for many rows of 16-bit operands on 16-byte boundaries: persistent warps walk over units of two rows x 256 columns, a row
// at a time with the next row's two loads in flight while one is computed; in the kernel above a thread loads, computes 20
// instructions per value and stores, one after another.  The lane that leads a block writes both rows' scales at once.  Cold
// operands, bf16, block 64, 11008 columns, kernel above against this one: 4096 rows 68.9 -> 54.7 us, 2048 36.5 -> 28.9, 1024 18.9 ->
// 15.7, 512 10.8 -> 9.0, 384 8.6 -> 8.6, 256 6.2 -> 5.4, 128 (2752 units) 4.05 -> 3.9, 64 (1376) 3.15 -> 3.2: kSiluWide lies between the
// last two.  Units of four rows: 2048 rows 30.4 us, 768 15.4 (the last round is emptier; 12.7 with two); of one row: 31.1 and 12.8.
// Four CTAs per SM instead of five (48 registers): 62.5 us against 60.4 with units of four; the exact silu out of line: 64.5 against 62.5.
constexpr int kSiluCtas = 5, kSiluRows = 2;
constexpr int64_t kSiluWide = 2500;

template <int QB, int DT>
__global__ void __launch_bounds__(kPreThreads, kSiluCtas) silu_mul_quantize_stream_kernel(const void* __restrict__ gate, const void* __restrict__ up,
                                                                               int64_t ldx, int8_t* __restrict__ q, int64_t ldq,
                                                                               float* __restrict__ sx, int M, int K, FastDiv col_units, unsigned units,
                                                                               int vec_s) {
    after_predecessor();
    constexpr int LPB = QB / 8;
    const int lane = threadIdx.x & 31;
    const unsigned warps = gridDim.x * (kPreThreads / 32);
    unsigned u = blockIdx.x * (kPreThreads / 32) + (threadIdx.x >> 5);
    if (u >= units) return;
    uint4 g, v;
    unsigned rg = col_units.div(u);
    int m = (int)rg * kSiluRows, k = (int)(u - rg * (unsigned)col_units.d) * 256 + lane * 8;
    auto fetch = [&](int row, int col) {
        g = v = make_uint4(0u, 0u, 0u, 0u);
        if (row < M && col < K) {
            const int64_t at = ((int64_t)row * ldx + col) * 2;
            g = ld_nc_v4(static_cast<const unsigned char*>(gate) + at);
            v = ld_nc_v4(static_cast<const unsigned char*>(up) + at);
        }
    };
    fetch(m, k);
    while (true) {
        const unsigned un = u + warps;
        int mn = M, kn = 0;
        if (un < units) {
            rg = col_units.div(un);
            mn = (int)rg * kSiluRows;
            kn = (int)(un - rg * (unsigned)col_units.d) * 256 + lane * 8;
        }
        float scale[kSiluRows];
#pragma unroll
        for (int r = 0; r < kSiluRows; ++r) {
            float y[8], w[8];
            {
                const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, vw[4] = {v.x, v.y, v.z, v.w};
                unpack8(y, gw, DT);
                unpack8(w, vw, DT);
            }
            if (r + 1 < kSiluRows) fetch(m + r + 1, k);
            else fetch(mn, kn);
            silu_mul8(y, w, DT);
            float amax = 0.0f;
#pragma unroll
            for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(y[e]));
#pragma unroll
            for (int off = 1; off < LPB; off <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
            scale[r] = amax;
            BlockQ bq;
            bq.set(amax, true);
            if (m + r < M && k < K) {
                uint32_t lo, hi;
                quantize8(y, bq, lo, hi);
                *reinterpret_cast<uint2*>(q + (int64_t)(m + r) * ldq + k) = make_uint2(lo, hi);
            }
        }
        if (lane % LPB == 0 && k < K) {
            float* dst = sx + (int64_t)(k / QB) * M + m;
            if (vec_s) {
                *reinterpret_cast<float2*>(dst) = make_float2(scale[0], scale[kSiluRows - 1]);
            } else {
#pragma unroll
                for (int r = 0; r < kSiluRows; ++r)
                    if (m + r < M) dst[r] = scale[r];
            }
        }
        if (un >= units) return;
        u = un;
        m = mn;
        k = kn;
    }
}

// C[m, n] = cast(C[m, n] + R[m, n]): the addition a layer's `x + proj(...)` performs in the activation type
__global__ void __launch_bounds__(kPreThreads) residual_add_kernel(void* C, int64_t ldc, const void* R, int64_t ldr, int dt, int64_t M,
                                                                   int64_t N) {
    after_predecessor();
    const int64_t i = (int64_t)blockIdx.x * kPreThreads + threadIdx.x;
    if (i >= M * N) return;
    const int64_t m = i / N, n = i % N, c = m * ldc + n, r = m * ldr + n;
    if (dt == BI8_F32) {
        static_cast<float*>(C)[c] = __fadd_rn(static_cast<float*>(C)[c], static_cast<const float*>(R)[r]);
    } else if (dt == BI8_BF16) {
        __nv_bfloat16* cp = static_cast<__nv_bfloat16*>(C);
        cp[c] = __float2bfloat16_rn(__fadd_rn(__bfloat162float(cp[c]), __bfloat162float(static_cast<const __nv_bfloat16*>(R)[r])));
    } else {
        __half* cp = static_cast<__half*>(C);
        cp[c] = __float2half_rn(__fadd_rn(__half2float(cp[c]), __half2float(static_cast<const __half*>(R)[r])));
    }
}

}  // namespace

int launch_residual_add(void* C, int64_t ldc, const void* R, int64_t ldr, int dt, int64_t M, int64_t N, cudaStream_t st) {
    if (M <= 0 || N <= 0) return BI8_OK;
    const int64_t blocks = (M * N + kPreThreads - 1) / kPreThreads;
    if (blocks > 0x7fffffff) return fail(BI8_ERR_LIMIT, "residual add: more than 2^31 blocks");
    return launch_chained(residual_add_kernel, (unsigned)blocks, kPreThreads, 0, st, C, ldc, R, ldr, dt, M, N);
}

int launch_quantize_pre(int op, const void* x, const void* x2, int dt, int64_t ldx, const void* weight, float eps, int8_t* q, int64_t ldq, float* sx,
                        int64_t M, int64_t K, int block, cudaStream_t st) {
    if (M == 0 || K == 0) return BI8_OK;
    if (M > 0x7fffffff || K > 0x3fffffff) return fail(BI8_ERR_LIMIT, "quantize_pre: M or K too large");
    const int esz = dt == BI8_F32 ? 4 : 2;
    const int nb = (int)((K + block - 1) / block);
    const bool rows16 = (ldx * esz) % 16 == 0 && K % 8 == 0;
    const int vec_in = rows16 && aligned(x, 16) && (!x2 || aligned(x2, 16)) && (!weight || aligned(weight, 16));
    const int vec_out = ldq % 8 == 0 && aligned(q, 8);
    if (op == BI8_PRE_NONE) return launch_quantize_rowwise(x, dt, ldx, q, ldq, sx, M, K, block, st);
    const int Mi = (int)M, Ki = (int)K;
    if (op == BI8_PRE_RMSNORM) {
        // 128 threads per row where the row fits their registers and there are rows enough to fill the SMs ten deep; a
        // handful of decode rows finish sooner with 256 threads each
        const bool narrow = (int64_t)nb * (block / 8) <= kPreHold * 128 && M > 1024;
        const int sms = device_info().sms;
        const bool early = !narrow && (int64_t)nb * (block / 8) <= kPreHold * 256 && (M <= 4 * sms || M > 5 * sms);
#define BI8_PRE_RMS_T(QB, T, EARLY)                                                                                                   \
    do {                                                                                                                             \
        if (dt == BI8_BF16) return launch_chained(rmsnorm_quantize_kernel<QB, T, BI8_BF16, EARLY>, (unsigned)M, T, 0, st, x, ldx, weight, eps, q, ldq, sx, Mi, Ki, nb, vec_in, vec_out); \
        else if (dt == BI8_F16) return launch_chained(rmsnorm_quantize_kernel<QB, T, BI8_F16, EARLY>, (unsigned)M, T, 0, st, x, ldx, weight, eps, q, ldq, sx, Mi, Ki, nb, vec_in, vec_out); \
        else return launch_chained(rmsnorm_quantize_kernel<QB, T, BI8_F32, false>, (unsigned)M, T, 0, st, x, ldx, weight, eps, q, ldq, sx, Mi, Ki, nb, vec_in, vec_out); \
    } while (0)
#define BI8_PRE_RMS(QB)                                                                                                              \
    if (narrow) BI8_PRE_RMS_T(QB, 128, false);                                                                                       \
    else if (early) BI8_PRE_RMS_T(QB, 256, true);                                                                                    \
    else BI8_PRE_RMS_T(QB, 256, false)
        switch (block) {
            case 32: BI8_PRE_RMS(32); break;
            case 64: BI8_PRE_RMS(64); break;
            case 128: BI8_PRE_RMS(128); break;
            default: return fail(BI8_ERR_BLOCK, "quantize_pre supports block 32, 64, 128 (got %d)", block);
        }
#undef BI8_PRE_RMS
#undef BI8_PRE_RMS_T
    } else if (op == BI8_PRE_SILU_MUL) {
        if (!x2) return fail(BI8_ERR_NULL, "quantize_pre: the gated activation needs its second operand");
        const int64_t units = M * nb * (block / 8);
        const unsigned grid = (unsigned)((units + kPreThreads - 1) / kPreThreads);
        const FastDiv upr((int64_t)nb * (block / 8));
        const int64_t col_units = (K + 255) / 256, wide = (M + kSiluRows - 1) / kSiluRows * col_units;
        if (dt != BI8_F32 && vec_in && vec_out && wide >= kSiluWide && wide < (1ll << 30)) {
            const FastDiv cu(col_units);
            const int vec_s = M % 2 == 0 && aligned(sx, 8);
            const int64_t want = (wide + kPreThreads / 32 - 1) / (kPreThreads / 32), fit = (int64_t)device_info().sms * kSiluCtas;
            const unsigned ctas = (unsigned)(want < fit || fit <= 0 ? want : fit);
#define BI8_PRE_SILU_STREAM(QB)                                                                                                      \
    if (block == QB) return dt == BI8_BF16 ? launch_chained(silu_mul_quantize_stream_kernel<QB, BI8_BF16>, ctas, kPreThreads, 0, st, x, x2, ldx, q, ldq, sx, Mi, Ki, cu, (unsigned)wide, vec_s) \
                                           : launch_chained(silu_mul_quantize_stream_kernel<QB, BI8_F16>, ctas, kPreThreads, 0, st, x, x2, ldx, q, ldq, sx, Mi, Ki, cu, (unsigned)wide, vec_s);
            BI8_PRE_SILU_STREAM(32) BI8_PRE_SILU_STREAM(64) BI8_PRE_SILU_STREAM(128)
#undef BI8_PRE_SILU_STREAM
        }
#define BI8_PRE_SILU(QB)                                                                                                             \
    do {                                                                                                                             \
        if (dt == BI8_BF16) return launch_chained(silu_mul_quantize_kernel<QB, BI8_BF16>, grid, kPreThreads, 0, st, x, x2, ldx, q, ldq, sx, Mi, Ki, upr, vec_in, vec_out); \
        else if (dt == BI8_F16) return launch_chained(silu_mul_quantize_kernel<QB, BI8_F16>, grid, kPreThreads, 0, st, x, x2, ldx, q, ldq, sx, Mi, Ki, upr, vec_in, vec_out); \
        else return launch_chained(silu_mul_quantize_kernel<QB, BI8_F32>, grid, kPreThreads, 0, st, x, x2, ldx, q, ldq, sx, Mi, Ki, upr, vec_in, vec_out); \
    } while (0)
        switch (block) {
            case 32: BI8_PRE_SILU(32); break;
            case 64: BI8_PRE_SILU(64); break;
            case 128: BI8_PRE_SILU(128); break;
            default: return fail(BI8_ERR_BLOCK, "quantize_pre supports block 32, 64, 128 (got %d)", block);
        }
#undef BI8_PRE_SILU
    } else {
        return fail(BI8_ERR_SHAPE, "quantize_pre: unknown operation code %d", op);
    }
    BI8_CUDA_TRY(cudaGetLastError());
    return BI8_OK;
}

}  // namespace bi8
