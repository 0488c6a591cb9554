// Block quantize / dequantize kernels (HBM-bound).
//
// Semantics follow the reference's kernels (paths inside the reference project):
//   quantize    triton_functions.py:382-406   scale = max|x| over the block (fp32),
//                                             q = rint(127 * (x / scale)), fp32 divide then fp32 multiply, RNE
//   dequantize  triton_functions.py:467-490   out = (scale * q) * fl32(1/127)
//   colwise     block_linear.py:93-94,100-103 transpose copy followed by the row-wise quantizer
//
// Data movement: every warp instruction of the vector kernels reads or writes one contiguous run of a
// row (32-byte or 16-byte per lane) and the block absmax is an xor-shuffle reduction inside the lanes that
// share a block.  The transposed scale tensor [K/block, rows] is written in 16-byte pieces (four rows of one
// block) by the streaming quantizer, and staged through shared memory by the tile kernels so that its
// stores (and, for dequantize, its loads) are contiguous along the row index.
#include "bi8_common.cuh"
#include "copy_rows.cuh"
#include "quant_math.cuh"
#include "tc_common.cuh"

#include <cstdlib>
#include <type_traits>

namespace bi8 {
namespace {

constexpr int kTileRows = 32;
constexpr int kThreads = 256;

__device__ __forceinline__ void ld_nc_v8(const void* p, uint32_t (&r)[8]) {
    asm volatile("ld.global.nc.L1::no_allocate.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "l"(p));
}
// ... and data that will not be read again: first in line to leave L2
__device__ __forceinline__ void ld_nc_far_v8(const void* p, uint32_t (&r)[8]) {
    asm volatile("ld.global.nc.L1::no_allocate.L2::evict_first.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "l"(p));
}
__device__ __forceinline__ void st_far_v8(void* p, const uint32_t (&r)[8]) {
    asm volatile("st.global.L2::evict_first.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void st_v8(void* p, const uint32_t (&r)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

template <typename T>
__device__ __forceinline__ float to_f32(T v);
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <>
__device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <>
__device__ __forceinline__ float to_f32<float>(float v) { return v; }

template <typename TO>
__device__ __forceinline__ TO from_f32(float v);
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <>
__device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }
template <>
__device__ __forceinline__ float from_f32<float>(float v) { return v; }

// two packed 16-bit floats -> two fp32
template <typename T>
__device__ __forceinline__ void unpack2(uint32_t w, float& lo, float& hi);
template <>
__device__ __forceinline__ void unpack2<__nv_bfloat16>(uint32_t w, float& lo, float& hi) {
    lo = bf16lo(w);
    hi = bf16hi(w);
}
template <>
__device__ __forceinline__ void unpack2<__half>(uint32_t w, float& lo, float& hi) {
    float2 f = __half22float2(*reinterpret_cast<__half2*>(&w));
    lo = f.x;
    hi = f.y;
}

// ------------------------------------------------------------------------------------------------
// Eight consecutive elements of a row as 4 or 8 words, from rows of any alignment.  The row is read in aligned 16-byte pieces:
// the `NW / 4` pieces that begin at or before the lane's first byte and, with SHIFT, the one behind them, and the words are
// funnel-shifted into place (the byte offset is the same in all lanes of a row, whose pieces are neighbours, so the
// repeated piece comes from L1).  A piece is read only where it contains a byte of the row, so no access leaves the
// tensor's 16-byte granules.  Elements from `valid` on read as zero.
template <typename T, bool SHIFT>
__device__ __forceinline__ void load_unit8(const T* p, const T* row_end, int valid, uint32_t (&w)[2 * sizeof(T)]) {
    constexpr int NW = 2 * (int)sizeof(T), NV = NW / 4;
    if constexpr (!SHIFT) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const uint4 d = ld_nc_v4(reinterpret_cast<const unsigned char*>(p) + 16 * v);
            w[4 * v] = d.x; w[4 * v + 1] = d.y; w[4 * v + 2] = d.z; w[4 * v + 3] = d.w;
        }
    } else {
        const uintptr_t a = reinterpret_cast<uintptr_t>(p), end = reinterpret_cast<uintptr_t>(row_end);
        const uintptr_t base = a & ~(uintptr_t)15;
        uint32_t r[NW + 4];
#pragma unroll
        for (int v = 0; v <= NV; ++v) {
            uint4 d = make_uint4(0u, 0u, 0u, 0u);
            if (base + 16 * v < end) d = __ldg(reinterpret_cast<const uint4*>(base + 16 * v));
            r[4 * v] = d.x; r[4 * v + 1] = d.y; r[4 * v + 2] = d.z; r[4 * v + 3] = d.w;
        }
        // the offset is the same in all lanes: a branch per word offset instead of selects per word
        const uint32_t off = (uint32_t)(a & 15u), bits = (off & 3u) * 8u;
        auto shifted = [&](auto words) {
            constexpr int WS = decltype(words)::value;
#pragma unroll
            for (int i = 0; i < NW; ++i) w[i] = __funnelshift_r(r[i + WS], r[i + WS + 1 < NW + 4 ? i + WS + 1 : NW + 3], bits);
        };
        if (off < 4u) shifted(std::integral_constant<int, 0>{});
        else if (off < 8u) shifted(std::integral_constant<int, 1>{});
        else if (off < 12u) shifted(std::integral_constant<int, 2>{});
        else shifted(std::integral_constant<int, 3>{});
    }
    if (valid < 8) {
#pragma unroll
        for (int i = 0; i < NW; ++i) {
            if constexpr (sizeof(T) == 4) {
                if (i >= valid) w[i] = 0u;
            } else {
                if (2 * i >= valid) w[i] = 0u;
                else if (2 * i + 1 >= valid) w[i] &= 0xffffu;
            }
        }
    }
}

// Row-wise quantize, vector path: any float type and (SHIFT) any alignment of the input rows; the int8 rows begin on 8-byte
// boundaries (pitch ldq).  A lane takes eight elements, a CTA covers 8 * RPW rows x 256 columns; warp w handles rows w, w+8,
// ... and issues their loads before any arithmetic.  RPW is 4, or 1 where that leaves SMs without a CTA: a row is eight
// divisions per lane in fp32, and four of them in sequence were 4.9 us of a 512 x 768 matrix's.  Bound by memory: for 16-bit inputs that the streaming kernel
// below does not take (rows that are not 32-byte aligned) and for fp32.
template <typename T, int B, bool SHIFT, int RPW>
__device__ __forceinline__ void quantize_rowwise_tile(int tile, const T* __restrict__ x, int64_t ldx, int8_t* __restrict__ q, int64_t ldq,
                                                      float* __restrict__ s, int M, int K, int nb, int col_tiles) {
    constexpr int WCOLS = 256;              // columns per warp pass
    constexpr int LPB = B / 8;              // lanes sharing one block
    constexpr int BPT = WCOLS / B;          // blocks per tile row
    constexpr int NW = 2 * (int)sizeof(T);  // 32-bit words of a lane's eight elements
    static_assert(LPB >= 1 && LPB <= 32, "block must be a multiple of the lane vector");
    constexpr int ROWS = 8 * RPW;
    __shared__ float s_scale[BPT][ROWS];

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ct = tile % col_tiles, rt = tile / col_tiles;
    const int col = ct * WCOLS + lane * 8;
    const int valid = K - col < 8 ? K - col : 8;          // elements of this lane inside the row; <= 0: none

    uint32_t raw[RPW][NW];
#pragma unroll
    for (int i = 0; i < RPW; ++i) {
        const int row = rt * ROWS + warp + 8 * i;
        if (valid > 0 && row < M) {
            const T* xr = x + (int64_t)row * ldx;
            load_unit8<T, SHIFT>(xr + col, xr + K, valid, raw[i]);
        } else {
#pragma unroll
            for (int w = 0; w < NW; ++w) raw[i][w] = 0u;
        }
    }
#pragma unroll
    for (int i = 0; i < RPW; ++i) {
        const int row = rt * ROWS + warp + 8 * i;
        float v[8];
        float amax = 0.0f;
        if constexpr (sizeof(T) == 4) {
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(raw[i][e]);
        } else {
#pragma unroll
            for (int w = 0; w < NW; ++w) unpack2<T>(raw[i][w], v[2 * w], v[2 * w + 1]);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(v[e]));
#pragma unroll
        for (int off = 1; off < LPB; off <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
        BlockQ bq;
        bq.set(amax, sizeof(T) == 2);
        uint32_t lo, hi;
        quantize8(v, bq, lo, hi);
        // a lane with fewer than eight elements writes zeros into the row's padding (ldq covers it: see the launcher)
        if (valid > 0 && row < M) *reinterpret_cast<uint2*>(q + (int64_t)row * ldq + col) = make_uint2(lo, hi);
        if ((lane % LPB) == 0) s_scale[lane / LPB][warp + 8 * i] = amax;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < BPT * ROWS; t += kThreads) {
        const int j = t / ROWS, r = t % ROWS;
        const int jb = ct * BPT + j, row = rt * ROWS + r;
        if (jb < nb && row < M) s[(int64_t)jb * M + row] = s_scale[j][r];
    }
}

template <typename T, int B, bool SHIFT, int RPW>
__global__ void __launch_bounds__(kThreads) quantize_rowwise_vec_kernel(
    const T* __restrict__ x, int64_t ldx, int8_t* __restrict__ q, int64_t ldq, float* __restrict__ s, int M, int K, int nb,
    int col_tiles) {
    after_predecessor();
    quantize_rowwise_tile<T, B, SHIFT, RPW>((int)blockIdx.x, x, ldx, q, ldq, s, M, K, nb, col_tiles);
}

// Row-wise quantize, streaming path (16-bit inputs, K % 16 == 0, 32-byte aligned rows).
// Persistent warps: a warp owns units of 4 rows x 512 columns (lane = 16 consecutive elements of a row, one
// 32-byte load and one 16-byte store per row) and keeps the loads of its NEXT unit in flight while it quantizes
// the current one, so the memory system always has 128 bytes per lane outstanding.  No shared memory and no CTA
// barrier: the lane that leads a block keeps the four row scales of its block and writes them as one 16-byte
// piece of the transposed scale tensor (s[j, m0..m0+3]).  The arithmetic is done on packed fp32 pairs.
// FAR: the input is too large to stay in L2 (kFarBytes) and leaves it first, so that the int8 result is still there for whoever
// reads it next (11008 x 4096 there and back: 48.1 -> 44.9 us with the dequantizer's stores treated alike).
template <typename T, int B, bool FAR>
__global__ void __launch_bounds__(kThreads, 2) quantize_rowwise_stream_kernel(
    const T* __restrict__ x, int64_t ldx, int8_t* __restrict__ q, int64_t ldq, float* __restrict__ s, int M, int K, int nb,
    FastDiv col_units, int64_t total_units) {
    after_predecessor();
    constexpr int LPB = B / 16;             // lanes sharing one block
    const int lane = threadIdx.x & 31;
    const int64_t gw = (int64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    const int64_t nw = (int64_t)gridDim.x * (kThreads / 32);
    // fl(127*y) and the round-to-integer step must stay two separately rounded operations.  A packed multiply
    // followed by a packed ADD was observed to come out as one fused operation (ties then round differently from
    // the reference's two-step evaluation), so the second step is written as fma(z, 1, magic): the product z*1 is
    // exact, the result is the single rounding of z + magic, and there is no multiply left to contract into it.
    const uint64_t c127 = f2_pack(127.0f, 127.0f), cmagic = f2_pack(kMagic, kMagic), cone = f2_pack(1.0f, 1.0f);
    auto round_pair = [&](uint64_t y2, uint32_t& b0, uint32_t& b1) {
        const uint64_t z = f2_mul(c127, y2);
        f2_bits(f2_fma(z, cone, cmagic), b0, b1);
    };

    auto row_group = [&](int64_t u) { return u < (1ll << 31) ? (int)col_units.div((unsigned)u) : (int)(u / col_units.d); };
    auto load_unit = [&](int64_t u, uint32_t (&buf)[4][8]) {
        const int rg = row_group(u), ct = (int)(u - (int64_t)rg * col_units.d);
        const int col = ct * 512 + lane * 16;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = rg * 4 + i;
            if (col < K && row < M) {
                if (FAR) ld_nc_far_v8(x + (int64_t)row * ldx + col, buf[i]);
                else ld_nc_v8(x + (int64_t)row * ldx + col, buf[i]);
            } else {
#pragma unroll
                for (int w = 0; w < 8; ++w) buf[i][w] = 0u;
            }
        }
    };
    auto process_unit = [&](int64_t u, const uint32_t (&buf)[4][8]) {
        const int rg = row_group(u), ct = (int)(u - (int64_t)rg * col_units.d);
        const int col = ct * 512 + lane * 16;
        float sc[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = rg * 4 + i;
            uint64_t v2[8];
            float amax = 0.0f;
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                float lo, hi;
                unpack2<T>(buf[i][w], lo, hi);
                amax = fmaxf(amax, fmaxf(fabsf(lo), fabsf(hi)));
                v2[w] = f2_pack(lo, hi);
            }
#pragma unroll
            for (int off = 1; off < LPB; off <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
            sc[i] = amax;
            BlockQ bq;
            bq.set(amax, true);
            uint32_t out[4];
            // bf16: `once` is `fast`; fp16 keeps the five operations.  Lanes behind the row's end have a scale of zero in every unit there: they
            // must not drag the warp through the divisions (3907 x 2688: 19.5 us for quantize and dequantize, 13.9 this way).
            constexpr bool ONCE = std::is_same_v<T, __nv_bfloat16>;
            if (ONCE && amax == 0.0f) {
#pragma unroll
                for (int w = 0; w < 4; ++w) out[w] = 0u;
            } else if (ONCE && bq.once) {
                const float r = bq.r127();
                const uint64_t r2 = f2_pack(r, r);
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    uint32_t b0, b1, b2, b3;
                    f2_bits(f2_fma(v2[2 * w], r2, cmagic), b0, b1);
                    f2_bits(f2_fma(v2[2 * w + 1], r2, cmagic), b2, b3);
                    out[w] = pack4(b0, b1, b2, b3);
                }
            } else if (!ONCE && bq.fast) {
                const uint64_t r2 = f2_pack(bq.rcp, bq.rcp), ns2 = f2_pack(-amax, -amax);
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    uint32_t b0, b1, b2, b3;
                    {
                        const uint64_t q0 = f2_mul(v2[2 * w], r2);
                        const uint64_t e = f2_fma(ns2, q0, v2[2 * w]);
                        const uint64_t y = f2_fma(e, r2, q0);
                        round_pair(y, b0, b1);
                    }
                    {
                        const uint64_t q0 = f2_mul(v2[2 * w + 1], r2);
                        const uint64_t e = f2_fma(ns2, q0, v2[2 * w + 1]);
                        const uint64_t y = f2_fma(e, r2, q0);
                        round_pair(y, b2, b3);
                    }
                    out[w] = pack4(b0, b1, b2, b3);
                }
            } else {
                if (ONCE) bq.fast = false;            // what is left are divisions
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    uint32_t a0, a1, a2, a3;
                    f2_bits(v2[2 * w], a0, a1);
                    f2_bits(v2[2 * w + 1], a2, a3);
                    out[w] = pack4(bq.q(__uint_as_float(a0)), bq.q(__uint_as_float(a1)), bq.q(__uint_as_float(a2)),
                                   bq.q(__uint_as_float(a3)));
                }
            }
            if (col < K && row < M)
                *reinterpret_cast<uint4*>(q + (int64_t)row * ldq + col) = make_uint4(out[0], out[1], out[2], out[3]);
        }
        if ((lane % LPB) == 0) {
            const int jb = (col / B);
            const int m0 = rg * 4;
            if (jb < nb && m0 < M) {
                float* dst = s + (int64_t)jb * M + m0;
                if (((M & 3) == 0)) {
                    *reinterpret_cast<float4*>(dst) = make_float4(sc[0], sc[1], sc[2], sc[3]);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (m0 + i < M) dst[i] = sc[i];
                }
            }
        }
    };

    uint32_t bufa[4][8], bufb[4][8];
    int64_t u = gw;
    if (u < total_units) load_unit(u, bufa);
    while (u < total_units) {
        const int64_t u1 = u + nw;
        if (u1 < total_units) load_unit(u1, bufb);
        process_unit(u, bufa);
        if (u1 >= total_units) break;
        const int64_t u2 = u1 + nw;
        if (u2 < total_units) load_unit(u2, bufa);
        process_unit(u1, bufb);
        u = u2;
    }
}

// Row-wise quantize to int8 rows that are not 8-byte aligned (a dense result whose row length is not a multiple of 8),
// block <= 64.  A warp takes kRagGroup consecutive blocks of one row; lane l handles elements l and l + 32 of every block, so
// all loads of the group (2-byte, coalesced) are in flight before the first absmax reduction, and the stores are runs of 32
// consecutive bytes.  Same arithmetic as every other quantizer (BlockQ).  What bounds it is a warp's chain of reductions: side by side
// instead of block after block 512 x 4100 takes 9.2 us (11.6), 4001 x 1001 13.9 (17.5), 300 x 777 4.6 (5.8); at block 32, with half the lanes idle, 13.0 (13.9).
constexpr int kRagGroup = 8;
template <typename T>
__global__ void __launch_bounds__(kThreads) quantize_rowwise_ragged_kernel(
    const T* __restrict__ x, int64_t ldx, int8_t* __restrict__ q, int64_t ldq, float* __restrict__ s, int64_t M, int64_t K, int B,
    int64_t nb, int64_t groups_per_row) {
    after_predecessor();
    const int lane = threadIdx.x & 31;
    const int64_t task = (int64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    if (task >= M * groups_per_row) return;
    const int64_t row = task / groups_per_row, j0 = (task % groups_per_row) * kRagGroup;
    const T* xr = x + row * ldx;
    float v[kRagGroup][2], amax[kRagGroup];
#pragma unroll
    for (int b = 0; b < kRagGroup; ++b) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int64_t k = (j0 + b) * B + lane + 32 * e;
            v[b][e] = (j0 + b < nb && lane + 32 * e < B && k < K) ? to_f32<T>(xr[k]) : 0.0f;
        }
    }
#pragma unroll
    for (int b = 0; b < kRagGroup; ++b) amax[b] = fmaxf(fabsf(v[b][0]), fabsf(v[b][1]));
    // the blocks' reductions side by side
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int b = 0; b < kRagGroup; ++b) amax[b] = fmaxf(amax[b], __shfl_xor_sync(0xffffffffu, amax[b], off));
#pragma unroll
    for (int b = 0; b < kRagGroup; ++b) {
        const int64_t j = j0 + b;
        if (j >= nb) break;
        BlockQ bq;
        bq.set(amax[b], sizeof(T) == 2);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int64_t k = j * B + lane + 32 * e;
            if (lane + 32 * e < B && k < K) q[row * ldq + k] = (int8_t)(bq.q(v[b][e]) & 0xffu);
        }
        if (lane == 0) s[j * M + row] = amax[b];
    }
}

// Row-wise quantize, any type / block / alignment: one warp per (row, block).
template <typename T>
__global__ void __launch_bounds__(kThreads) quantize_rowwise_generic_kernel(
    const T* __restrict__ x, int64_t ldx, int8_t* __restrict__ q, int64_t ldq, float* __restrict__ s, int64_t M, int64_t K, int B,
    int64_t nb) {
    after_predecessor();
    const int lane = threadIdx.x & 31;
    const int64_t task = (int64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    if (task >= M * nb) return;
    const int64_t row = task / nb, j = task % nb;
    const int64_t lo = j * B, hi = (lo + B < K) ? lo + B : K;
    const T* xr = x + row * ldx;
    float amax = 0.0f;
    for (int64_t k = lo + lane; k < hi; k += 32) amax = fmaxf(amax, fabsf(to_f32<T>(xr[k])));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    BlockQ bq;
    bq.set(amax, sizeof(T) == 2);
    for (int64_t k = lo + lane; k < hi; k += 32) q[row * ldq + k] = (int8_t)(bq.q(to_f32<T>(xr[k])) & 0xffu);
    if (lane == 0) s[j * M + row] = amax;
}

// ------------------------------------------------------------------------------------------------
// Column-wise quantize for fp32 inputs and for 16-bit ones that the tile quantizer does not take.  A CTA takes one block of B
// rows x 64 columns: a thread has one column and B/4 consecutive rows, all of whose loads are in flight before the
// first absmax; the four row groups of a column exchange their maxima through shared memory, the bytes go to a
// transposed tile, and each column's B bytes leave as 16-byte pieces (bytes where the output is not aligned).  With one thread per column
// and a loop down the block (the kernel below) a 300 x 256 matrix took 9 us of serial loads.
template <typename T, int B>
__device__ __forceinline__ void quantize_colwise_tile(int tile_index, const T* __restrict__ x, int64_t ldx, int8_t* __restrict__ q, int64_t ldq,
                                                      float* __restrict__ s, int R, int C, int col_tiles) {
    constexpr int TC = 64, GROUPS = kThreads / TC, RPT = B / GROUPS;     // columns, row groups, rows per thread
    constexpr int PITCH = B + 16;                                        // bytes; rows 16-byte aligned
    __shared__ float s_max[GROUPS][TC];
    __shared__ __align__(16) unsigned char tile[TC * PITCH];
    const int j = tile_index / col_tiles, c0 = (tile_index % col_tiles) * TC;
    const int c = threadIdx.x % TC, g = threadIdx.x / TC;
    const int r0 = j * B + g * RPT;
    const bool col_ok = c0 + c < C;
    const T* xc = x + (int64_t)r0 * ldx + c0 + c;
    float v[RPT];
    float amax = 0.0f;
#pragma unroll
    for (int r = 0; r < RPT; ++r) v[r] = (col_ok && r0 + r < R) ? to_f32<T>(xc[(int64_t)r * ldx]) : 0.0f;
#pragma unroll
    for (int r = 0; r < RPT; ++r) amax = fmaxf(amax, fabsf(v[r]));
    s_max[g][c] = amax;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < GROUPS; ++k) amax = fmaxf(amax, s_max[k][c]);
    BlockQ bq;
    bq.set(amax, sizeof(T) == 2);
    if (g == 0 && col_ok) s[(int64_t)j * C + c0 + c] = amax;
#pragma unroll
    for (int r = 0; r < RPT; r += 4)
        *reinterpret_cast<uint32_t*>(tile + c * PITCH + g * RPT + r) = pack4(bq.q(v[r]), bq.q(v[r + 1]), bq.q(v[r + 2]), bq.q(v[r + 3]));
    __syncthreads();
    constexpr int PIECES = B / 16;
    const bool vec = (ldq & 15) == 0 && (reinterpret_cast<uintptr_t>(q) & 15u) == 0;
    for (int t = threadIdx.x; t < TC * PIECES; t += kThreads) {
        const int cc = t / PIECES, rr = (t % PIECES) * 16, left = R - (j * B + rr);
        if (c0 + cc >= C || left <= 0) continue;
        const unsigned char* src = tile + cc * PITCH + rr;
        int8_t* dst = q + (int64_t)(c0 + cc) * ldq + j * B + rr;
        if (vec && left >= 16) {
            *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(src);
        } else {
            for (int b = 0; b < 16 && b < left; ++b) dst[b] = (int8_t)src[b];
        }
    }
}

template <typename T, int B>
__global__ void __launch_bounds__(kThreads) quantize_colwise_cols_kernel(
    const T* __restrict__ x, int64_t ldx, int8_t* __restrict__ q, int64_t ldq, float* __restrict__ s, int R, int C, int col_tiles) {
    after_predecessor();
    quantize_colwise_tile<T, B>((int)blockIdx.x, x, ldx, q, ldq, s, R, C, col_tiles);
}

// Column-wise quantize for the other block sizes, rows of any alignment.  A CTA takes
// one block of B rows x kThreads columns: thread t reads its column down the block twice (absmax, then quantize; the
// second pass hits L1/L2; consecutive threads read consecutive columns), parks the B bytes in shared memory, and the
// warps then write each output row's B bytes as runs of 32 consecutive bytes.  (With one thread storing its column byte
// by byte, every warp store touched 32 sectors.)  Dynamic shared memory: kThreads * (B + 4) bytes.
template <typename T>
__global__ void __launch_bounds__(kThreads) quantize_colwise_ragged_kernel(
    const T* __restrict__ x, int64_t ldx, int8_t* __restrict__ q, int64_t ldq, float* __restrict__ s, int64_t R, int64_t C, int B,
    int64_t col_tiles) {
    after_predecessor();
    extern __shared__ unsigned char tile[];                 // [kThreads][B + 4]
    const int pitch = B + 4;
    const int64_t j = blockIdx.x / col_tiles, c0 = (blockIdx.x % col_tiles) * kThreads;
    const int64_t lo = j * B;
    const int rows = (int)((lo + B < R) ? B : R - lo);
    const int64_t c = c0 + threadIdx.x;
    if (c < C) {
        const T* xc = x + lo * ldx + c;
        float amax = 0.0f;
        for (int r = 0; r < rows; ++r) amax = fmaxf(amax, fabsf(to_f32<T>(xc[(int64_t)r * ldx])));
        BlockQ bq;
        bq.set(amax, sizeof(T) == 2);
        unsigned char* mine = tile + (size_t)threadIdx.x * pitch;
        for (int r = 0; r < rows; ++r) mine[r] = (unsigned char)(bq.q(to_f32<T>(xc[(int64_t)r * ldx])) & 0xffu);
        s[j * C + c] = amax;
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int t = warp; t < kThreads; t += kThreads / 32) {
        const int64_t cc = c0 + t;
        if (cc >= C) break;
        int8_t* dst = q + cc * ldq + lo;
        const unsigned char* src = tile + (size_t)t * pitch;
        for (int r = lane; r < rows; r += 32) dst[r] = (int8_t)src[r];
    }
}

// Column-wise quantize, any type / block / alignment: one thread per (block, column).
template <typename T>
__global__ void __launch_bounds__(kThreads) quantize_colwise_generic_kernel(
    const T* __restrict__ x, int64_t ldx, int8_t* __restrict__ q, int64_t ldq, float* __restrict__ s, int64_t R, int64_t C, int B,
    int64_t nb) {
    after_predecessor();
    const int64_t task = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (task >= nb * C) return;
    const int64_t j = task / C, c = task % C;
    const int64_t lo = j * B, hi = (lo + B < R) ? lo + B : R;
    float amax = 0.0f;
    for (int64_t r = lo; r < hi; ++r) amax = fmaxf(amax, fabsf(to_f32<T>(x[r * ldx + c])));
    BlockQ bq;
    bq.set(amax, sizeof(T) == 2);
    for (int64_t r = lo; r < hi; ++r) q[c * ldq + r] = (int8_t)(bq.q(to_f32<T>(x[r * ldx + c])) & 0xffu);
    s[j * C + c] = amax;
}

// ------------------------------------------------------------------------------------------------
// Dequantize, vector path: a lane owns 16 consecutive int8 (one 16-byte load) and writes 16 outputs.
// The CTA tile is 32 rows x 512 columns; its scales [512/B][32] are loaded row-contiguously first.
// (FAR: the output is too large to stay in L2 and must not push the int8 rows out that are still to be read.)
template <bool FAR, typename TO>
__device__ __forceinline__ void store16(TO* o, const float (&f)[16]) {
    uint32_t w[16];
#pragma unroll
    for (int i = 0; i < (sizeof(TO) == 4 ? 16 : 8); ++i) {
        if constexpr (std::is_same_v<TO, float>) w[i] = __float_as_uint(f[i]);
        else if constexpr (std::is_same_v<TO, __half>) w[i] = pack_f16x2(f[2 * i], f[2 * i + 1]);
        else w[i] = pack_bf16x2(f[2 * i], f[2 * i + 1]);
    }
#pragma unroll
    for (int h = 0; h < (sizeof(TO) == 4 ? 2 : 1); ++h) {
        const uint32_t r[8] = {w[8 * h], w[8 * h + 1], w[8 * h + 2], w[8 * h + 3], w[8 * h + 4], w[8 * h + 5], w[8 * h + 6], w[8 * h + 7]};
        if (FAR) st_far_v8(reinterpret_cast<uint32_t*>(o) + 8 * h, r);
        else st_v8(reinterpret_cast<uint32_t*>(o) + 8 * h, r);
    }
}

template <typename TO, int B, bool FAR>
__global__ void __launch_bounds__(kThreads) dequantize_rowwise_vec_kernel(
    const int8_t* __restrict__ q, int64_t ldq, const float* __restrict__ s, TO* __restrict__ out, int M, int K, int nb,
    int col_tiles) {
    after_predecessor();
    constexpr int WCOLS = 512;
    constexpr int BPT = WCOLS / B;
    constexpr int LPB = B / 16;
    __shared__ float s_scale[BPT][kTileRows];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ct = blockIdx.x % col_tiles, rt = blockIdx.x / col_tiles;
    const int col = ct * WCOLS + lane * 16;
    const bool col_ok = col < K;            // K % 16 == 0 on this path

    uint4 raw[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int row = rt * kTileRows + warp + 8 * i;
        raw[i] = (col_ok && row < M) ? ld_nc_v4(q + (int64_t)row * ldq + col) : make_uint4(0u, 0u, 0u, 0u);
    }
    for (int t = threadIdx.x; t < BPT * kTileRows; t += kThreads) {
        const int j = t / kTileRows, r = t % kTileRows;
        const int jb = ct * BPT + j, row = rt * kTileRows + r;
        s_scale[j][r] = (jb < nb && row < M) ? s[(int64_t)jb * M + row] : 0.0f;
    }
    __syncthreads();
    const float inv127 = 1.0f / 127.0f;     // fl32(1/127), the constant the reference passes (line 499)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int row = rt * kTileRows + warp + 8 * i;
        if (!(col_ok && row < M)) continue;
        const float sc = s_scale[lane / LPB][warp + 8 * i];
        const uint32_t w[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
        float f[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            const int v = (int)(int8_t)((w[e / 4] >> (8 * (e % 4))) & 0xffu);
            f[e] = __fmul_rn(__fmul_rn(sc, (float)v), inv127);
        }
        store16<FAR>(out + (int64_t)row * K + col, f);
    }
}

// Dequantize to rows that are not 32-byte aligned (K not a multiple of 16), or any block size and alignment.  A warp takes a
// run of 256 columns of a row; a lane's four stores are aligned 4-byte words (two 16-bit results, or one fp32), 32 lanes
// next to each other, whatever the row's alignment: for a 16-bit row that begins between two words, the words hold elements
// (2i - 1, 2i) and the row's first and last element are stored alone.
template <typename TO>
__global__ void __launch_bounds__(kThreads) dequantize_rowwise_words_kernel(
    const int8_t* __restrict__ q, int64_t ldq, const float* __restrict__ s, TO* __restrict__ out, int64_t M, int K, int B, int log2_b, int col_units) {
    after_predecessor();
    constexpr int EPW = 4 / (int)sizeof(TO), WORDS = 256 / (32 * EPW);   // elements per word, words per lane
    const int lane = threadIdx.x & 31;
    const int64_t unit = (int64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    const int64_t m = unit / col_units;
    if (m >= M) return;
    TO* row = out + m * K;
    const int odd = (int)((reinterpret_cast<uintptr_t>(row) & 3u) / sizeof(TO));    // elements past a word boundary: 0 or 1
    const int first = (int)(unit % col_units) * 256 - odd;
    const int8_t* qr = q + m * ldq;
    const float inv127 = 1.0f / 127.0f;
    int8_t b[WORDS][EPW];
    float sc[WORDS][EPW];
#pragma unroll
    for (int w = 0; w < WORDS; ++w)
#pragma unroll
        for (int e = 0; e < EPW; ++e) {
            const int k = first + (w * 32 + lane) * EPW + e;
            const bool in = k >= 0 && k < K;
            b[w][e] = in ? qr[k] : (int8_t)0;
            const int j = log2_b >= 0 ? k >> log2_b : k / B;
            sc[w][e] = in ? __ldg(s + (int64_t)j * M + m) : 0.0f;
        }
#pragma unroll
    for (int w = 0; w < WORDS; ++w) {
        const int k = first + (w * 32 + lane) * EPW;
        TO v[EPW];
#pragma unroll
        for (int e = 0; e < EPW; ++e) v[e] = from_f32<TO>(__fmul_rn(__fmul_rn(sc[w][e], (float)b[w][e]), inv127));
        if (k >= 0 && k + EPW <= K) {
            uint32_t word;
            if constexpr (EPW == 1) word = __float_as_uint(v[0]);
            else word = (uint32_t)*reinterpret_cast<const uint16_t*>(&v[0]) | ((uint32_t)*reinterpret_cast<const uint16_t*>(&v[EPW - 1]) << 16);
            *reinterpret_cast<uint32_t*>(row + k) = word;
        } else {
#pragma unroll
            for (int e = 0; e < EPW; ++e)
                if (k + e >= 0 && k + e < K) row[k + e] = v[e];
        }
    }
}

// Several small jobs of one pass in one launch: row-wise and column-wise quantizations, column sums, copies of int8 rows to aligned
// ones.  For matrices of a few hundred KB each of them is a launch (2 to 3 us of host time and as much latency on the device) around
// well under a microsecond of work.  A CTA finds its job by its index; the tiles are those of the single-purpose kernels.
enum JobKind { kJobRow = 0, kJobRowShift, kJobCol, kJobSum, kJobCopy };
struct Job {
    const void* x;
    void* q;            // int8 result; kJobSum: the sums
    float* s;
    int64_t ldx, ldq;
    int M, K, nb, tiles, kind, end;       // `end`: first CTA of the next job
};
constexpr int kMostJobs = 8;
struct Jobs {
    Job job[kMostJobs];
};

// Sums of 32 columns over all rows by eight groups of rows, added in the groups' order (fp32).
template <typename T>
__device__ __forceinline__ void column_sum_tile(int tile, const T* __restrict__ x, int64_t ldx, T* __restrict__ out, int R, int C) {
    __shared__ float part[8][32];
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5, c = tile * 32 + lane;
    const int per = (R + 7) / 8, r1 = (g + 1) * per < R ? (g + 1) * per : R;
    float acc = 0.0f;
    if (c < C) {
        int r = g * per;
        for (; r + 8 <= r1; r += 8) {
            float f[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) f[u] = to_f32<T>(x[(int64_t)(r + u) * ldx + c]);
#pragma unroll
            for (int u = 0; u < 8; ++u) acc += f[u];
        }
        for (; r < r1; ++r) acc += to_f32<T>(x[(int64_t)r * ldx + c]);
    }
    part[g][lane] = acc;
    __syncthreads();
    if (g == 0 && c < C) {
        float v = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) v += part[k][lane];
        out[c] = from_f32<T>(v);
    }
}

template <typename T, int B>
__global__ void __launch_bounds__(kThreads) quantize_jobs_kernel(const __grid_constant__ Jobs jobs) {
    after_predecessor();
    int k = 0;
    while ((int)blockIdx.x >= jobs.job[k].end) ++k;
    const Job& j = jobs.job[k];
    const int tile = (int)blockIdx.x - (k ? jobs.job[k - 1].end : 0);
    const T* x = static_cast<const T*>(j.x);
    int8_t* q = static_cast<int8_t*>(j.q);
    if (j.kind == kJobRow) quantize_rowwise_tile<T, B, false, 1>(tile, x, j.ldx, q, j.ldq, j.s, j.M, j.K, j.nb, j.tiles);
    else if (j.kind == kJobRowShift) quantize_rowwise_tile<T, B, true, 1>(tile, x, j.ldx, q, j.ldq, j.s, j.M, j.K, j.nb, j.tiles);
    else if (j.kind == kJobCol) quantize_colwise_tile<T, B>(tile, x, j.ldx, q, j.ldq, j.s, j.M, j.K, j.tiles);
    else if (j.kind == kJobSum) column_sum_tile<T>(tile, x, j.ldx, static_cast<T*>(j.q), j.M, j.K);
    else copy_rows_piece((int64_t)tile * kThreads + threadIdx.x, static_cast<const int8_t*>(j.x), j.ldx, q, j.ldq, (int64_t)j.M * j.tiles, j.tiles, j.K);
}

// From here on a tensor and what is computed from it do not both stay in L2 (126 MB).
constexpr int64_t kFarBytes = 64 << 20;

bool use_v8() {
    static const bool on = (std::getenv("BI8_NO_V8") == nullptr);
    return on;
}

template <typename T>
int quantize_rowwise_t(const T* x, int64_t ldx, int8_t* q, int64_t ldq, float* s, int64_t M, int64_t K, int block, cudaStream_t st) {
    const int64_t nb = (K + block - 1) / block;
    const bool small = M < (1ll << 31) && K < (1ll << 30);
    const bool block_ok = block == 32 || block == 64 || block == 128 || block == 256;
    if constexpr (sizeof(T) == 2) {
        if (small && use_v8() && K % 16 == 0 && ldx % 16 == 0 && aligned(x, 32) && ldq % 16 == 0 && aligned(q, 16) && aligned(s, 16) && block_ok) {
            const DeviceInfo di = device_info();
            const int col_units = (int)((K + 511) / 512);
            const int64_t total = ((M + 3) / 4) * col_units;
            int64_t ctas = (total + kThreads / 32 - 1) / (kThreads / 32);   // one unit per warp at least
            if (ctas > 2ll * di.sms) ctas = 2ll * di.sms;                   // two resident CTAs per SM, persistent beyond that
            auto launch = [&](auto kernel) {
                return launch_chained(kernel, (unsigned)ctas, kThreads, 0, st, x, ldx, q, ldq, s, (int)M, (int)K, (int)nb, FastDiv(col_units), total);
            };
            const bool far = M * K * (int64_t)sizeof(T) > kFarBytes;
#define BI8_QSTREAM(BB) \
    if (block == BB) return far ? launch(quantize_rowwise_stream_kernel<T, BB, true>) : launch(quantize_rowwise_stream_kernel<T, BB, false>);
            BI8_QSTREAM(32) BI8_QSTREAM(64) BI8_QSTREAM(128) BI8_QSTREAM(256)
#undef BI8_QSTREAM
        }
    }
    // Any input alignment, as long as the int8 rows are 8-byte aligned and their pitch covers a lane's last eight elements.
    const int64_t ctiles = (K + 255) / 256;
    const bool few = ((M + 31) / 32) * ctiles < 2ll * device_info().sms;
    const int64_t row_tiles = few ? (M + 7) / 8 : (M + 31) / 32;
    if (small && block_ok && ldq % 8 == 0 && aligned(q, 8) && row_tiles * ctiles < (1ll << 31)) {
        const bool straight = K % 8 == 0 && aligned(x, 16) && (ldx * (int64_t)sizeof(T)) % 16 == 0;
        auto launch = [&](auto kernel) {
            return launch_chained(kernel, (unsigned)(row_tiles * ctiles), kThreads, 0, st, x, ldx, q, ldq, s, (int)M, (int)K, (int)nb, (int)ctiles);
        };
#define BI8_QROW(BB)                                                                                                              \
    if (block == BB && few)                                                                                                       \
        return straight ? launch(quantize_rowwise_vec_kernel<T, BB, false, 1>) : launch(quantize_rowwise_vec_kernel<T, BB, true, 1>); \
    if (block == BB)                                                                                                              \
        return straight ? launch(quantize_rowwise_vec_kernel<T, BB, false, 4>) : launch(quantize_rowwise_vec_kernel<T, BB, true, 4>);
        BI8_QROW(32) BI8_QROW(64) BI8_QROW(128) BI8_QROW(256)
#undef BI8_QROW
    }
    if (block <= 64) {
        const int64_t gpr = (nb + kRagGroup - 1) / kRagGroup;
        const int64_t rgrid = (M * gpr + kThreads / 32 - 1) / (kThreads / 32);
        if (rgrid < (1ll << 31))
            return launch_chained(quantize_rowwise_ragged_kernel<T>, (unsigned)rgrid, kThreads, 0, st, x, ldx, q, ldq, s, M, K, block, nb, gpr);
    }
    const int64_t tasks = M * nb;
    const int64_t grid = (tasks + kThreads / 32 - 1) / (kThreads / 32);
    if (grid >= (1ll << 31)) return fail(BI8_ERR_SHAPE, "quantize_rowwise: %lld blocks exceed the grid limit", (long long)tasks);
    return launch_chained(quantize_rowwise_generic_kernel<T>, (unsigned)grid, kThreads, 0, st, x, ldx, q, ldq, s, M, K, block, nb);
}

template <typename T>
int quantize_colwise_t(const T* x, int64_t ldx, int8_t* q, int64_t ldq, float* s, int64_t R, int64_t C, int block, cudaStream_t st) {
    const bool small = R < (1ll << 31) - 256 && C < (1ll << 31) - 256;
    const int64_t nb = (R + block - 1) / block;
    const int64_t ctiles = (C + 63) / 64;
    if (small && nb * ctiles < (1ll << 31)) {
        const unsigned grid = (unsigned)(nb * ctiles);
#define BI8_QCOLS(BB) \
    if (block == BB) return launch_chained(quantize_colwise_cols_kernel<T, BB>, grid, kThreads, 0, st, x, ldx, q, ldq, s, (int)R, (int)C, (int)ctiles);
        BI8_QCOLS(32) BI8_QCOLS(64) BI8_QCOLS(128)
#undef BI8_QCOLS
    }
    if (block <= 256) {
        const int64_t col_tiles = (C + kThreads - 1) / kThreads;
        const size_t smem = (size_t)kThreads * (block + 4);
        if (nb * col_tiles < (1ll << 31)) {
            if (smem > 48 * 1024) {
                static SmemOptIn opt_in;
                const int rc = opt_in.ensure(quantize_colwise_ragged_kernel<T>, smem);
                if (rc != BI8_OK) return rc;
            }
            return launch_chained(quantize_colwise_ragged_kernel<T>, (unsigned)(nb * col_tiles), kThreads, smem, st, x, ldx, q, ldq, s, R, C, block, col_tiles);
        }
    }
    const int64_t grid = (nb * C + kThreads - 1) / kThreads;
    if (grid >= (1ll << 31)) return fail(BI8_ERR_SHAPE, "quantize_colwise: grid too large");
    return launch_chained(quantize_colwise_generic_kernel<T>, (unsigned)grid, kThreads, 0, st, x, ldx, q, ldq, s, R, C, block, nb);
}

template <typename TO>
int dequantize_t(const int8_t* q, int64_t ldq, const float* s, TO* out, int64_t M, int64_t K, int block, cudaStream_t st) {
    const int64_t nb = (K + block - 1) / block;
    const bool small = M < (1ll << 31) && K < (1ll << 30);
    const int64_t row_tiles = (M + kTileRows - 1) / kTileRows, ctiles = (K + 511) / 512;
    if (small && use_v8() && K % 16 == 0 && ldq % 16 == 0 && aligned(q, 16) && aligned(out, 32) && row_tiles * ctiles < (1ll << 31)) {
        auto launch = [&](auto kernel) {
            return launch_chained(kernel, (unsigned)(row_tiles * ctiles), kThreads, 0, st, q, ldq, s, out, (int)M, (int)K, (int)nb, (int)ctiles);
        };
        const bool far = M * K * (int64_t)sizeof(TO) > kFarBytes;
#define BI8_DEQ(BB) \
    if (block == BB) return far ? launch(dequantize_rowwise_vec_kernel<TO, BB, true>) : launch(dequantize_rowwise_vec_kernel<TO, BB, false>);
        BI8_DEQ(32) BI8_DEQ(64) BI8_DEQ(128) BI8_DEQ(256)
#undef BI8_DEQ
    }
    const int64_t units = (K + 1 + 255) / 256;              // one element more: a row may begin between two words
    const int64_t grid = (M * units + kThreads / 32 - 1) / (kThreads / 32);
    if (grid >= (1ll << 31) || K >= (1ll << 30)) return fail(BI8_ERR_SHAPE, "dequantize: grid too large");
    int log2_b = -1;
    for (int i = 0; i < 31; ++i)
        if (block == (1 << i)) log2_b = i;
    return launch_chained(dequantize_rowwise_words_kernel<TO>, (unsigned)grid, kThreads, 0, st, q, ldq, s, out, M, (int)K, block, log2_b, (int)units);
}

}  // namespace

int launch_quantize_rowwise(const void* x, int dt, int64_t ldx, int8_t* q, int64_t ldq, float* s, int64_t M, int64_t K, int block,
                            cudaStream_t st) {
    switch (dt) {
        case BI8_BF16: return quantize_rowwise_t(static_cast<const __nv_bfloat16*>(x), ldx, q, ldq, s, M, K, block, st);
        case BI8_F16: return quantize_rowwise_t(static_cast<const __half*>(x), ldx, q, ldq, s, M, K, block, st);
        case BI8_F32: return quantize_rowwise_t(static_cast<const float*>(x), ldx, q, ldq, s, M, K, block, st);
    }
    return fail(BI8_ERR_DTYPE, "quantize_rowwise: unknown dtype code %d", dt);
}

int launch_quantize_colwise(const void* x, int dt, int64_t ldx, int8_t* q, int64_t ldq, float* s, int64_t R, int64_t C, int block,
                            cudaStream_t st) {
    if (quantize_tile_applicable(dt, q, ldq, nullptr, 0, R, C, block))
        return launch_quantize_tile(x, dt, ldx, q, ldq, s, nullptr, 0, nullptr, R, C, block, st);
    switch (dt) {
        case BI8_BF16: return quantize_colwise_t(static_cast<const __nv_bfloat16*>(x), ldx, q, ldq, s, R, C, block, st);
        case BI8_F16: return quantize_colwise_t(static_cast<const __half*>(x), ldx, q, ldq, s, R, C, block, st);
        case BI8_F32: return quantize_colwise_t(static_cast<const float*>(x), ldx, q, ldq, s, R, C, block, st);
    }
    return fail(BI8_ERR_DTYPE, "quantize_colwise: unknown dtype code %d", dt);
}

int launch_dequantize_rowwise(const int8_t* q, int64_t ldq, const float* s, void* out, int dt, int64_t M, int64_t K, int block,
                              cudaStream_t st) {
    switch (dt) {
        case BI8_BF16: return dequantize_t(q, ldq, s, static_cast<__nv_bfloat16*>(out), M, K, block, st);
        case BI8_F16: return dequantize_t(q, ldq, s, static_cast<__half*>(out), M, K, block, st);
        case BI8_F32: return dequantize_t(q, ldq, s, static_cast<float*>(out), M, K, block, st);
    }
    return fail(BI8_ERR_DTYPE, "dequantize: unknown dtype code %d", dt);
}

// The most values that a launch of several jobs quantizes (row-wise and column-wise counted each), and the most int8 values that it copies
// beside them: up to there it takes no longer on the device than the single-purpose kernels one after another (a training step's
// quantizers at 2048 x 768 x 768, 4.3 M in the forward pass with separate kernels 16.9 us, at 1024 x 512 x 512 15.6 -> 8.8) and is two
// or three launches of 2 to 3 us of host time less: 300 x 256 x 384 in fp32 99 -> 82 us a step, 11 launches -> 5, 512 x 1024 x
// 1024 bf16 91 -> 81; a layer of 333 x 1000 x 777 with unaligned weights 13.6 -> 12.3 us.  Column sums of more than kJobSumRows
// rows want more CTAs than a job gives them.
namespace {
constexpr int64_t kJobValues = 4 << 20, kJobCopied = 1 << 20;
constexpr int kJobSumRows = 512;

// One launch's worth of jobs, or a negative number where some task needs a kernel of its own.
int collect_jobs(const bi8_quantize_task* t, int n, int block, Jobs* jobs) {
    if (block != 32 && block != 64 && block != 128) return -1;
    int count = 0, dt = -1;
    int64_t values = 0, ctas = 0;
    for (int i = 0; i < n; ++i) {
        const bi8_quantize_task& a = t[i];
        if (a.rows <= 0 || a.cols <= 0 || a.rows >= (1 << 30) || a.cols >= (1 << 30)) return -1;
        auto add = [&](int kind, const void* x, void* q, int64_t ldq, float* s, int nb, int tiles, int64_t blocks) {
            if (count == kMostJobs) return false;
            ctas += blocks;
            if (ctas >= (1ll << 30)) return false;
            if (jobs) jobs->job[count] = Job{x, q, s, a.ldx, ldq, (int)a.rows, (int)a.cols, nb, tiles, kind, (int)ctas};
            ++count;
            return true;
        };
        if (a.x_dtype == BI8_I8) {
            const int64_t per_row = (a.cols + 15) / 16;
            if (a.rows * a.cols > kJobCopied || a.q_col || a.sum || !add(kJobCopy, a.x, a.q_row, a.ldq_row, nullptr, 0, (int)per_row, (a.rows * per_row + kThreads - 1) / kThreads)) return -1;
            continue;
        }
        if (dt >= 0 && dt != a.x_dtype) return -1;
        dt = a.x_dtype;
        values += a.rows * a.cols * ((a.q_row ? 1 : 0) + (a.q_col ? 1 : 0));
        const int esz = dt == BI8_F32 ? 4 : 2;
        if (a.q_row) {
            if (a.ldq_row % 8 != 0 || !aligned(a.q_row, 8)) return -1;
            const int64_t ctiles = (a.cols + 255) / 256;
            const bool straight = a.cols % 8 == 0 && aligned(a.x, 16) && a.ldx * esz % 16 == 0;
            if (!add(straight ? kJobRow : kJobRowShift, a.x, a.q_row, a.ldq_row, a.s_row, (int)((a.cols + block - 1) / block), (int)ctiles, (a.rows + 7) / 8 * ctiles)) return -1;
        }
        if (a.q_col) {
            const int64_t ctiles = (a.cols + 63) / 64;
            if (!add(kJobCol, a.x, a.q_col, a.ldq_col, a.s_col, 0, (int)ctiles, (a.rows + block - 1) / block * ctiles)) return -1;
        }
        if (a.sum) {
            if (a.rows > kJobSumRows || !add(kJobSum, a.x, a.sum, 0, nullptr, 0, 0, (a.cols + 31) / 32)) return -1;
        }
    }
    return dt >= 0 && values <= kJobValues ? count : -1;
}

template <typename T>
int launch_jobs(const Jobs& jobs, int count, int block, cudaStream_t st) {
    const unsigned ctas = (unsigned)jobs.job[count - 1].end;
    return block == 32   ? launch_chained(quantize_jobs_kernel<T, 32>, ctas, kThreads, 0, st, jobs)
           : block == 64 ? launch_chained(quantize_jobs_kernel<T, 64>, ctas, kThreads, 0, st, jobs)
                         : launch_chained(quantize_jobs_kernel<T, 128>, ctas, kThreads, 0, st, jobs);
}
}  // namespace

bool quantize_jobs_fit(const bi8_quantize_task* tasks, int n, int block) { return collect_jobs(tasks, n, block, nullptr) > 1; }

int launch_quantize_jobs(const bi8_quantize_task* tasks, int n, int block, cudaStream_t st) {
    Jobs jobs{};
    const int count = collect_jobs(tasks, n, block, &jobs);
    if (count < 1) return fail(BI8_ERR_LIMIT, "quantize_many: the tasks do not fit one launch");
    int dt = BI8_I8;
    for (int i = 0; i < n; ++i)
        if (tasks[i].x_dtype != BI8_I8) dt = tasks[i].x_dtype;
    return dt == BI8_BF16 ? launch_jobs<__nv_bfloat16>(jobs, count, block, st) : dt == BI8_F16 ? launch_jobs<__half>(jobs, count, block, st) : launch_jobs<float>(jobs, count, block, st);
}

}  // namespace bi8
