// Int8 block GEMM with fused dequantize for few activation rows (decode and small batches: M <= 64), on the sm_100a tensor
// cores with the operand roles exchanged.
//
// Same contract as the reference kernel at triton_functions.py:69-139 (path inside the reference project).  With so few
// rows of A the work is one pass over the weights Bt[N, K]: the kernel is bound by streaming them from HBM, and is
// organised around that stream and around the fixed cost of a call, which is as long as the stream itself for a 4096 x 4096
// matrix.
//   * The weights are the M operand of the MMA: a tile is 128 weight rows, the activations (padded to 16, 32 or 64
//     rows) are the N operand, so one tcgen05.mma kind::i8 (M128 N16..64 K32) covers 128 weight rows and every
//     activation row, and the s32 accumulator of a quantisation block is only 16..64 tensor-memory columns.
//   * Clusters of 1, 2, 4 or 8 CTAs work on a tile together, each on its share of K (split_plan: whatever lets the
//     most SMs stream for the fewest stages), one CTA per SM; clusters walk over the tiles.  The partial sums of
//     a tile meet in shared memory of the cluster: quarter q of the tile's rows is finished by CTA q mod cluster size,
//     the others send theirs with st.async, which counts its bytes on the receiver's mbarrier, and the receiver
//     adds them in ascending K order.  One kernel, no workspace, and the exchange costs about half a microsecond.  (Equal
//     ranges of a stream-K sequence with a second kernel for the sums keep all 148 SMs streaming but need a
//     launch more, 2.3 us of host time; sums inside the kernel through L2, by flags or by self-describing pieces, cost
//     2 us of device time per call: a store, a poll and the cold code are one L2 trip each.)
//   * Activations either arrive quantized (SRC 0) or are quantized by the kernel itself (SRC 1, M <= 32): every CTA takes the
//     rows' share of K that its own stages need (with the RMSNorm or SiLU * mul step in front, if asked for) and leaves it in
//     shared memory as the MMA's swizzled operand tiles, while the first weights are on their way.  That is one launch
//     and one kernel boundary less per layer; the redundancy (every cluster quantizes the same rows) is hidden behind
//     the weights' first arrival only where a CTA's part is short.  Where it is not (kQuantInKernelValues in api.cu has the line
//     and both sides) and above 16 rows they come from skinny_quantize_kernel or one of the producer
//     quantizers, launched in front so that this kernel's set-up and first weight copies overlap them.
//   * Warp roles: promotion warps (four per 16 activation rows, or per 32 for 64 rows; one per tensor-memory lane
//     quarter) convert and scale; one producer warp issues, per stage, the TMA copies that complete on one
//     barrier: 128 weight rows x 128 K-bytes, the stage's weight scales (a [blocks, 128] fp32 box of sB) and, with SRC 0,
//     the activation rows of the same K range; two MMA issuer warps take the stages in turn (one accumulator range per
//     quantisation block, one commit per stage); with SRC 1 five more warps help to quantize.
//   * Promotion follows the reference's order term by term, sB*(sA*(float(P)*fl32(1/127^2))), added in ascending block
//     order within a CTA's share of K, so a tile that is not divided is bit-identical to the CUDA-core kernel.
#include "quant_math.cuh"
#include "tc_common.cuh"
#include "peer_common.cuh"

#include <cstring>

namespace bi8 {
namespace {

using namespace ptx;

constexpr int kTileRows = 128;    // weight rows per tile (the MMA's M)
constexpr int kSkMaxM = 64;       // beyond 64 activation rows the promotion (5 instructions per element and block, in the
                                  // reference's order) costs more than the weights take to arrive: measured slower than
                                  // the general kernel at 128 rows
constexpr int kMostCluster = 8;   // the portable limit

constexpr int pow2_at_least(int x) {
    int p = 32;
    while (p < x) p *= 2;
    return p;
}

constexpr int kHelpWarps = 5;     // SRC 1: warps that only quantize (512 threads: 128 registers each)

template <int QB, int BNS, int SRC>
struct SkGeo {
    // A stage is SUB operand tiles of 128 K-bytes: what a stage costs beside its bytes (barrier hand-overs, a commit, the
    // tensor-memory round trip) is about 400 cycles per role, as long as 128 x 128 bytes take to arrive.
    static constexpr int SUB = BNS <= 32 ? 2 : 1;
    static constexpr int KS = SUB * kBK;                  // K bytes of a stage
    static constexpr int STAGES = BNS == 16 ? (SRC == 0 ? 5 : 4) : BNS == 32 ? (SRC == 0 ? 4 : 3) : 5;
    static constexpr int BPS = KS / QB;                   // quantisation blocks per stage
    static constexpr int MMAS = QB / 32;                  // MMAs (K = 32) per block
    static constexpr int CW = BNS / 2;                    // activation rows (accumulator columns) per promotion warp
    static constexpr int CHUNKS = BNS / CW;
    static constexpr int PROMO_WARPS = 4 * CHUNKS;
    static constexpr int VB = BPS * CW <= 32 ? BPS : 32 / CW;      // blocks whose accumulators a promotion thread loads at once
    static constexpr int ACC_STRIDE = BPS * BNS;          // tensor-memory columns of one stage's accumulators
    static constexpr int NBUF = (512 / ACC_STRIDE) < 4 || STAGES < 4 ? 2 : 4;     // no more than there are stages: see the MMA issuers
    static constexpr int MMA_WARPS = 2;                   // MMA issuers, taking the stages in turn
    static constexpr int THREADS = (PROMO_WARPS + 1 + MMA_WARPS + (SRC != 0 ? kHelpWarps : 0)) * 32;
    static constexpr int TMEM_COLS = pow2_at_least(NBUF * ACC_STRIDE);
    static constexpr uint32_t W_BYTES = SUB * kTileRows * kBK;
    static constexpr uint32_t XT_BYTES = BNS * kBK;                       // one operand tile of activations (128 K-bytes)
    static constexpr uint32_t X_BYTES = SRC == 0 ? SUB * XT_BYTES : 0;    // ... inside a stage
    static constexpr uint32_t S_TX = BPS * kTileRows * 4;                 // bytes the scale copy delivers
    static constexpr uint32_t S_BYTES = S_TX < 1024 ? 1024 : S_TX;        // keeps every stage 1024-byte aligned
    static constexpr uint32_t STAGE_BYTES = W_BYTES + X_BYTES + S_BYTES;
    static constexpr uint32_t bar_off = STAGES * STAGE_BYTES;
    static_assert(NBUF % MMA_WARPS == 0 && VB >= 1 && BPS % VB == 0, "every issuer keeps its own accumulators; whole groups of blocks");
    static constexpr int FULL_AB = 0, EMPTY_AB = STAGES, ACC_FULL = 2 * STAGES, ACC_EMPTY = 2 * STAGES + NBUF,
                         RX_FULL = 2 * STAGES + 2 * NBUF,                 // [2 buffers][promotion warps]: parts have arrived
                         RX_FREE = RX_FULL + 2 * PROMO_WARPS,             // [2 buffers][promotion warps]: the receiver is done with ours
                         NBARS = RX_FREE + 2 * PROMO_WARPS;
    static constexpr uint32_t misc_off = bar_off + NBARS * 8;             // tmem holder, abort flag, never-raised flag
    static constexpr uint32_t norm_off = (misc_off + 32 + 15) & ~15u;     // SRC 1, RMSNorm: sums of squares [BNS][8]
    static constexpr uint32_t rx_off = norm_off + (SRC != 0 ? BNS * 8 * 4 : 0);   // received parts, see rx_bytes()
};

struct SkParams {
    const float* sA;
    const void* X;          // SRC 1: activations before quantization, row pitch ldx elements
    const void* X2;         // SRC 1: second operand of SiLU * mul (same pitch), or the RMSNorm weight, or null
    int64_t ldx;
    float eps;
    int x_dtype, op;
    const void* bias;
    int64_t bias_ld;        // row pitch of `bias` in elements: 0 = one row for all (a bias), else an [M, N] addend (a residual)
    void* C;
    int* status;
    int64_t ldc;
    int M, N, K, nb, nks, tiles;
    int out_dtype, bias_dtype;
    int live_chunks;    // groups of CW activation rows that hold a valid row
    int early_weights;  // the weight copies of the first stages may be issued before the preceding kernel has completed
    int rx_bufs;        // receive buffers: 2 where a cluster has more than one tile
    int share;          // most stages of a CTA
    uint32_t sx_off, xq_off;    // activation scales [share * BPS][BNS]; SRC 1: operand tiles [share * SUB][BNS x 128 bytes]
};

// Bytes of one receive buffer: for every quarter this CTA finishes and every CTA of the cluster, 32 rows x BNS sums.
__host__ __device__ constexpr uint32_t rx_bytes(int bns, int cluster) {
    return (uint32_t)(cluster == 1 ? 0 : cluster * (cluster < 4 ? 4 / cluster : 1) * 32 * bns * 4);
}

// dynamic shared memory of a launch, and where its run-time sized parts begin
template <int QB, int BNS, int SRC>
size_t smem_of(int share, int cluster, int rx_bufs, uint32_t* sx_off = nullptr, uint32_t* xq_off = nullptr) {
    using G = SkGeo<QB, BNS, SRC>;
    const uint32_t sx = G::rx_off + (uint32_t)rx_bufs * rx_bytes(BNS, cluster);
    uint32_t end = sx + (uint32_t)(share * G::BPS * BNS * 4);
    if (sx_off) *sx_off = sx;
    if (SRC != 0) {
        end = (end + 1023u) & ~1023u;
        if (xq_off) *xq_off = end;
        end += (uint32_t)(share * G::SUB) * G::XT_BYTES;
    }
    return (size_t)end + 1024;                            // alignment slack
}

// ---- cluster helpers ----------------------------------------------------------------------------------------------------
// 16 bytes into another CTA's shared memory, counted there on `cluster_bar`
__device__ __forceinline__ void send_v4(uint32_t cluster_addr, uint32_t cluster_bar, float a, float b, float c, float d) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%2, %3, %4, %5}, [%1];" ::"r"(cluster_addr),
                 "r"(cluster_bar), "f"(a), "f"(b), "f"(c), "f"(d)
                 : "memory");
}
// ---- output -------------------------------------------------------------------------------------------------------------
// C[m, n] = cast(acc) (+ cast(addend) in the output type: reference lines 125-131) for the CW rows of a chunk and one column n; the
// addend is bias[n] (bias_ld 0) or an [M, N] residual.  All addends are requested before the first is used.
template <typename T>
__device__ __forceinline__ T round_as(float v);
template <>
__device__ __forceinline__ __nv_bfloat16 round_as<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <>
__device__ __forceinline__ __half round_as<__half>(float v) { return __float2half_rn(v); }
template <>
__device__ __forceinline__ float round_as<float>(float v) { return v; }
__device__ __forceinline__ float widen(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float widen(__half v) { return __half2float(v); }
__device__ __forceinline__ float widen(float v) { return v; }

template <typename T>
__device__ __forceinline__ void finish_rows(const float* acc, const float (&add)[8], bool has_add, int live, T* c, int64_t ldc) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (i >= live) break;
        T v = round_as<T>(acc[i]);
        if (has_add) v = round_as<T>(__fadd_rn(widen(v), widen(round_as<T>(add[i]))));
        c[(int64_t)i * ldc] = v;
    }
}

template <int CW>
__device__ __forceinline__ void finish_chunk(const float (&acc)[CW], const SkParams& p, int m0, int n) {
#pragma unroll
    for (int g = 0; g < CW; g += 8) {
        const int m = m0 + g, live = p.M - m < 8 ? p.M - m : 8;
        if (live <= 0) break;
        float add[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) add[i] = 0.0f;
        const bool has_add = p.bias != nullptr;
        if (has_add) {
            const int64_t b0 = (int64_t)m * p.bias_ld + n;
            if (p.bias_dtype == BI8_F32) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (i < live) add[i] = static_cast<const float*>(p.bias)[b0 + i * p.bias_ld];
            } else {
                unsigned short h[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) h[i] = i < live ? static_cast<const unsigned short*>(p.bias)[b0 + i * p.bias_ld] : (unsigned short)0;
#pragma unroll
                for (int i = 0; i < 8; ++i) add[i] = p.bias_dtype == BI8_BF16 ? bf16lo(h[i]) : __half2float(__ushort_as_half(h[i]));
            }
        }
        const int64_t o = (int64_t)m * p.ldc + n;
        if (p.out_dtype == BI8_BF16) finish_rows(acc + g, add, has_add, live, static_cast<__nv_bfloat16*>(p.C) + o, p.ldc);
        else if (p.out_dtype == BI8_F16) finish_rows(acc + g, add, has_add, live, static_cast<__half*>(p.C) + o, p.ldc);
        else finish_rows(acc + g, add, has_add, live, static_cast<float*>(p.C) + o, p.ldc);
    }
}

// ---- quantization inside the kernel (SRC 1) ------------------------------------------------------------------------------
// eight consecutive elements of a 16-byte aligned row: request, and conversion of what has arrived
struct Raw8 {
    uint4 a, b;           // b: the second half of eight fp32 values
};
__device__ __forceinline__ Raw8 request_x8(const void* base, int64_t index, int dt) {
    Raw8 r;
    if (dt == BI8_F32) {
        const float* src = static_cast<const float*>(base) + index;
        r.a = ld_nc_v4(src);
        r.b = ld_nc_v4(src + 4);
    } else {
        r.a = ld_nc_v4(static_cast<const unsigned short*>(base) + index);
        r.b = make_uint4(0u, 0u, 0u, 0u);
    }
    return r;
}
__device__ __forceinline__ void convert_x8(float (&f)[8], const Raw8& r, int dt) {
    if (dt == BI8_F32) {
        f[0] = __uint_as_float(r.a.x); f[1] = __uint_as_float(r.a.y); f[2] = __uint_as_float(r.a.z); f[3] = __uint_as_float(r.a.w);
        f[4] = __uint_as_float(r.b.x); f[5] = __uint_as_float(r.b.y); f[6] = __uint_as_float(r.b.z); f[7] = __uint_as_float(r.b.w);
    } else {
        const uint32_t w4[4] = {r.a.x, r.a.y, r.a.z, r.a.w};
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
}

// The activations' share [k0, k1) of 128-byte K steps, by `warps` whole warps (this one is `me`): producer step, block scales into
// sx [block][BNS], int8 values into the MMA's operand tiles (128-byte swizzle: the 16-byte chunk index is xor-ed with the row
// index mod 8) at shared address xq.  Values, scales and the order of RMSNorm's sum are those of the stand-alone quantizers
// (quantize_pre.cu at 256 threads per row).  Elements from K on are not written: the weights' zero fill meets them.
// All loads of a batch are requested before the first is used: the whole step is a few trips to L2, in front of which the
// weights wait.
template <int QB, int BNS>
__device__ __forceinline__ void quantize_share(const SkParams& p, int k0, int k1, int me, int warps, int lane, float* norm, float* sx, uint32_t xq) {
    constexpr int LPB = QB / 8;
    const int dt = p.x_dtype;
    if (p.op == BI8_PRE_RMSNORM) {
        // sums of squares of whole rows: 256 virtual threads per row, a warp plays 32 of them at a time, four times at once
        constexpr int TASKS = 4;
        const int tasks = p.M * 8, steps = (p.K + 2047) / 2048;
        for (int t0 = me; t0 < tasks; t0 += warps * TASKS) {
            float ss[TASKS] = {0.0f, 0.0f, 0.0f, 0.0f};
            for (int i = 0; i < steps; ++i) {
                Raw8 r[TASKS];
#pragma unroll
                for (int q = 0; q < TASKS; ++q) {
                    const int t = t0 + q * warps, k = i * 2048 + ((t & 7) * 32 + lane) * 8;
                    r[q].a = r[q].b = make_uint4(0u, 0u, 0u, 0u);
                    if (t < tasks && k < p.K) r[q] = request_x8(p.X, (int64_t)(t >> 3) * p.ldx + k, dt);
                }
#pragma unroll
                for (int q = 0; q < TASKS; ++q) {
                    float f[8];
                    convert_x8(f, r[q], dt);
#pragma unroll
                    for (int e = 0; e < 8; ++e) ss[q] = __fmaf_rn(f[e], f[e], ss[q]);
                }
            }
#pragma unroll
            for (int q = 0; q < TASKS; ++q) {
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) ss[q] += __shfl_xor_sync(0xffffffffu, ss[q], off);
                if (lane == 0 && t0 + q * warps < tasks) norm[t0 + q * warps] = ss[q];
            }
        }
        asm volatile("bar.sync 3, %0;" ::"r"(warps * 32) : "memory");
    }
    const int upr = (k1 - k0) * (kBK / 8);                 // units of eight elements per row
    const int units = p.M * upr;
    constexpr int BATCH = 4;
    for (int u0 = me * 32; u0 < units; u0 += warps * 32 * BATCH) {     // upr is a multiple of 16: a block's lanes stay together
        Raw8 rx[BATCH], r2[BATCH];
#pragma unroll
        for (int q = 0; q < BATCH; ++q) {
            const int u = u0 + q * warps * 32 + lane, m = u / upr, k = k0 * kBK + (u - m * upr) * 8;
            rx[q].a = rx[q].b = r2[q].a = r2[q].b = make_uint4(0u, 0u, 0u, 0u);
            if (u < units && k < p.K) {
                rx[q] = request_x8(p.X, (int64_t)m * p.ldx + k, dt);
                if (p.op == BI8_PRE_SILU_MUL) r2[q] = request_x8(p.X2, (int64_t)m * p.ldx + k, dt);
                else if (p.op == BI8_PRE_RMSNORM && p.X2 != nullptr) r2[q] = request_x8(p.X2, k, dt);
            }
        }
#pragma unroll
        for (int q = 0; q < BATCH; ++q) {
            if (u0 + q * warps * 32 >= units) break;
            const int u = u0 + q * warps * 32 + lane, m = u / upr, piece = u - m * upr, k = k0 * kBK + piece * 8;
            const bool valid = u < units && k < p.K;
            float f[8];
            convert_x8(f, rx[q], dt);
            if (p.op != BI8_PRE_NONE && valid) {
                float v[8];
                convert_x8(v, r2[q], dt);
                if (p.op == BI8_PRE_SILU_MUL) {
                    silu_mul8(f, v, dt);
                } else {
                    float total = 0.0f;
#pragma unroll
                    for (int w = 0; w < 8; ++w) total += norm[m * 8 + w];
                    const float rstd = rsqrtf(__fadd_rn(__fdiv_rn(total, (float)p.K), p.eps));
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        float y = __fmul_rn(f[e], rstd);
                        if (p.X2) y = __fmul_rn(y, v[e]);
                        f[e] = round_to(y, dt);
                    }
                }
            }
            float amax = 0.0f;
#pragma unroll
            for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(f[e]));
#pragma unroll
            for (int off = 1; off < LPB; off <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
            if (!valid) continue;
            BlockQ bq;
            bq.set(amax, dt != BI8_F32);
            uint32_t lo, hi;
            quantize8(f, bq, lo, hi);
            const int tile = piece / (kBK / 8), c16 = piece % (kBK / 8);
            const uint32_t dst = xq + (uint32_t)(tile * BNS * kBK + m * 128 + ((((c16 >> 1) ^ (m & 7)) << 4) | ((c16 & 1) << 3)));
            asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(dst), "r"(lo), "r"(hi) : "memory");
            if ((piece % LPB) == 0) sx[(piece / LPB) * BNS + m] = amax;
        }
    }
}

template <int QB, int BNS, int SRC>
__global__ void __launch_bounds__(SkGeo<QB, BNS, SRC>::THREADS, 1)
gemm_tc_skinny_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                      const __grid_constant__ CUtensorMap tmS, const SkParams p) {
    using G = SkGeo<QB, BNS, SRC>;
    constexpr int CW = G::CW;
    extern __shared__ __align__(1024) unsigned char smem_dyn[];
    const uint32_t raw = smem_u32(smem_dyn);
    const uint32_t base = (raw + 1023u) & ~1023u;      // the swizzle atom needs 1024-byte alignment (the same in every CTA)
    unsigned char* base_ptr = smem_dyn + (base - raw);
    const uint32_t bars = base + G::bar_off;
    volatile uint32_t* tmem_holder = reinterpret_cast<volatile uint32_t*>(base_ptr + G::misc_off);
    const uint32_t abort_flag = base + G::misc_off + 4;
    const uint32_t never_flag = base + G::misc_off + 8;
    float* sx = reinterpret_cast<float*>(base_ptr + p.sx_off);
    const uint32_t sx_u32 = base + p.sx_off;
    auto bar = [&](int slot) -> uint32_t { return bars + 8u * (uint32_t)slot; };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int live_warps = 4 * p.live_chunks;
    constexpr int PW = G::PROMO_WARPS, MW = G::PROMO_WARPS + 1;

    // this CTA's place: rank `rank` of `CL` in its cluster, K stages [k0, k1) of every tile; the cluster takes tiles
    // first_tile, first_tile + tile_step, ...
    const int CL = (int)cluster_size(), rank = (int)cluster_rank();
    const int first_tile = (int)blockIdx.x / CL, tile_step = (int)gridDim.x / CL;
    const int k0 = rank * p.nks / CL, k1 = (rank + 1) * p.nks / CL, len = k1 - k0;
    const int rounds = first_tile < p.tiles ? (p.tiles - first_tile + tile_step - 1) / tile_step : 0;
    const int my_stages = rounds * len;

    auto issue_x = [&](int stage, int ks) {
#pragma unroll
        for (int u = 0; u < G::SUB; ++u)
            tma_load_2d(base + (uint32_t)stage * G::STAGE_BYTES + G::W_BYTES + (uint32_t)u * G::XT_BYTES, &tmX, bar(G::FULL_AB + stage),
                        ks * G::KS + u * kBK, 0);
    };
    // one lane; `with_x` false leaves out the activation tile, whose copy then has to follow (issue_x)
    auto issue_stage = [&](int stage, int tile, int ks, bool with_x) {
        const uint32_t dst = base + (uint32_t)stage * G::STAGE_BYTES;
        mbar_expect_tx(bar(G::FULL_AB + stage), G::W_BYTES + G::X_BYTES + G::S_TX);
#pragma unroll
        for (int u = 0; u < G::SUB; ++u)
            tma_load_2d(dst + (uint32_t)(u * kTileRows * kBK), &tmW, bar(G::FULL_AB + stage), ks * G::KS + u * kBK, tile * kTileRows);
        if (SRC == 0 && with_x) issue_x(stage, ks);
        tma_load_2d(dst + G::W_BYTES + G::X_BYTES, &tmS, bar(G::FULL_AB + stage), tile * kTileRows, ks * G::BPS);
    };

    // The producer warp sets the barriers up, tells the others (named barrier 2: it arrives, they wait, so it never stands
    // still) and starts the copies of the first stages right away: the ring is empty, nothing has to be waited for.  The
    // tensor-memory allocation runs beside it.
    int pre_tile = first_tile, pre_ks = k0, pre_count = 0;
    if (warp == PW) {
        if (lane == 0) {
            for (int s = 0; s < G::STAGES; ++s) {
                mbar_init(bar(G::FULL_AB + s), 1);                             // the TMA's bytes
                // a stage is free again when every promotion warp has seen its accumulator complete (so the MMAs have
                // read the operands) and has taken its scales
                mbar_init(bar(G::EMPTY_AB + s), live_warps);
            }
            for (int b = 0; b < G::NBUF; ++b) {
                mbar_init(bar(G::ACC_FULL + b), 1);
                mbar_init(bar(G::ACC_EMPTY + b), live_warps);
            }
            for (int b = 0; b < 2 * PW; ++b) {
                mbar_init(bar(G::RX_FULL + b), 1);
                mbar_init(bar(G::RX_FREE + b), 1);
            }
            sts_u32(abort_flag, 0u);
            sts_u32(never_flag, 0u);
            mbar_fence_init();
            fence_proxy_async_smem();
        }
        __syncwarp();
        asm volatile("bar.arrive 2, %0;" ::"n"(G::THREADS) : "memory");
        cluster_arrive();                                                      // barriers are set up: see the first send
        // The kernel is always launched so that it may start before its predecessor in the stream has completed.  Behind
        // this library's own activation quantizer the weights are known to be at rest and their copies start at once;
        // behind any other kernel (which may be the one writing the weights) nothing is read before the wait.
        if (!p.early_weights) after_predecessor();
        else asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        while (pre_count < G::STAGES && pre_count < my_stages) {
            if (elect_one()) issue_stage(pre_count, pre_tile, pre_ks, false);
            ++pre_count;
            if (++pre_ks == k1) { pre_ks = k0; pre_tile += tile_step; }
        }
        // Everything above touched only the weights and their scales.  The activations come from the kernel launched just
        // before this one (a quantizer that lets its dependents start early): wait for it here.
        if (p.early_weights) asm volatile("griddepcontrol.wait;" ::: "memory");
        if (SRC == 0 && elect_one()) {
            int ks = k0;
            for (int q = 0; q < pre_count; ++q) {
                issue_x(q, ks);
                if (++ks == k1) ks = k0;
            }
        }
        __syncwarp();
    }
    if (warp == MW) {
        tmem_alloc(smem_u32((const void*)tmem_holder), G::TMEM_COLS);
        tmem_relinquish();
    }
    if (warp != PW) {
        tc_fence_before();
        asm volatile("bar.sync 2, %0;" ::"n"(G::THREADS) : "memory");
        cluster_arrive();
        tc_fence_after();
        asm volatile("griddepcontrol.wait;" ::: "memory");      // activations, their scales, and every store, after the previous kernel
    }
    const uint32_t tmem_base = (warp != PW) ? *tmem_holder : 0u;       // the producer never touches tensor memory
    bool cluster_ready = false;                                        // this thread has waited for the cluster's set-up

    if (SRC != 0 && warp != PW) {
        // every warp but the producer quantizes; the generic stores are handed to the tensor core's proxy before the barrier
        constexpr int QWARPS = G::THREADS / 32 - 1;
        quantize_share<QB, BNS>(p, k0 * G::SUB, k1 * G::SUB, warp < PW ? warp : warp - 1, QWARPS, lane, reinterpret_cast<float*>(base_ptr + G::norm_off), sx,
                                base + p.xq_off);
        fence_proxy_async_smem();
        asm volatile("bar.sync 3, %0;" ::"n"(QWARPS * 32) : "memory");
    }

    if (warp == PW) {
        // ---------------- TMA producer ----------------
        int stage = pre_count == G::STAGES ? 0 : pre_count;
        uint32_t phase = pre_count == G::STAGES ? 1u : 0u;
        int last_parity[G::STAGES];
#pragma unroll
        for (int q = 0; q < G::STAGES; ++q) last_parity[q] = q < pre_count ? 0 : -1;
        int tile = pre_tile, ks = pre_ks;
        bool ok = true;
        for (int s = pre_count; s < my_stages; ++s) {
            ok = __all_sync(0xffffffffu, mbar_wait(bar(G::EMPTY_AB + stage), phase ^ 1u, abort_flag));
            if (!ok) {
                if (lane == 0) report_timeout(p.status, abort_flag, W_EMPTY_AB);
                break;
            }
            if (elect_one()) issue_stage(stage, tile, ks, true);
            __syncwarp();
#pragma unroll
            for (int q = 0; q < G::STAGES; ++q)
                if (q == stage) last_parity[q] = (int)phase;
            if (++stage == G::STAGES) { stage = 0; phase ^= 1u; }
            if (++ks == k1) { ks = k0; tile += tile_step; }
        }
        if (!ok) {
            // do not leave while our own copies may still land in this CTA's shared memory
#pragma unroll
            for (int q = 0; q < G::STAGES; ++q)
                if (last_parity[q] >= 0) (void)mbar_wait(bar(G::FULL_AB + q), (uint32_t)last_parity[q], never_flag, 200000000ll);
        }
        __syncwarp();
    } else if (warp >= MW && warp < MW + G::MMA_WARPS) {
        // ---------------- MMA issuers ----------------
        // Issuing the MMAs of a stage, the commit and the polls of its two barriers cost one thread several hundred cycles, so
        // MMA_WARPS warps take the stages in turn.
        static_assert(G::MMA_WARPS <= G::STAGES, "an issuer advances by at most one turn of the stage ring");
        static_assert(G::STAGES % G::MMA_WARPS == 0 || G::NBUF <= G::STAGES, "see the waits below");
        constexpr uint32_t idesc = umma_idesc_i8(kTileRows, BNS);
        // One elected thread runs the loop (as in the general kernel): no votes, and no lane picked out around every issue.  In a graph, with
        // the producer's issues and the promotion warps' releases alike: decode layer of 8 sequences (4096, 11008) 64.0 -> 63.1 us, one row
        // through 4096 x 4096 6.44 -> 6.24.
        if (elect_one()) {
            const int me = warp - MW;
            int buf = me, stage = me, ks = me;               // ks: stage inside this CTA's share
            while (len > 0 && ks >= len) ks -= len;
            uint32_t phase = 0, accphase = 0;
            for (int s = me; s < my_stages; s += G::MMA_WARPS) {
                // An accumulator range is free, then the operands have landed.  The order matters where the number of
                // stages is odd and a stage's uses alternate between the issuers: a parity wait also succeeds while the use before
                // the awaited one is still under way, and that use is known to be over only because its accumulators (at most
                // NBUF <= STAGES uses back) have been read.
                const bool got_acc = mbar_wait(bar(G::ACC_EMPTY + buf), accphase ^ 1u, abort_flag);
                if (!got_acc || !mbar_wait(bar(G::FULL_AB + stage), phase, abort_flag)) {
                    report_timeout(p.status, abort_flag, got_acc ? W_FULL_AB : W_ACC_EMPTY);
                    break;
                }
                tc_fence_after();
                const uint32_t st_base = base + (uint32_t)stage * G::STAGE_BYTES;
                const uint64_t wdesc = umma_desc_k_sw128(st_base);
                const uint64_t xdesc = umma_desc_k_sw128(SRC == 0 ? st_base + G::W_BYTES : base + p.xq_off + (uint32_t)(ks * G::SUB) * G::XT_BYTES);
#pragma unroll
                for (int blk = 0; blk < G::BPS; ++blk) {
                    if ((k0 + ks) * G::BPS + blk < p.nb) {
#pragma unroll
                        for (int i = 0; i < G::MMAS; ++i) {
                            const int kb = (blk * G::MMAS + i) * 32, sub = kb / kBK;           // K byte inside the stage, operand tile
                            const uint64_t koff = (uint64_t)(kb % kBK / 16);
                            mma_i8(tmem_base + (uint32_t)(buf * G::ACC_STRIDE + blk * BNS), wdesc + koff + (uint64_t)(sub * kTileRows * kBK / 16),
                                   xdesc + koff + (uint64_t)(sub * (int)G::XT_BYTES / 16), idesc, i > 0 ? 1u : 0u);
                        }
                    }
                }
                // one commit per stage: the promotion warps release the stage's shared memory once they have seen it
                tc_commit(bar(G::ACC_FULL + buf));
                stage += G::MMA_WARPS;
                if (stage >= G::STAGES) { stage -= G::STAGES; phase ^= 1u; }
                buf += G::MMA_WARPS;
                if (buf >= G::NBUF) { buf -= G::NBUF; accphase ^= 1u; }
                ks += G::MMA_WARPS;
                while (ks >= len) ks -= len;
            }
        }
        __syncwarp();
    } else if (warp < PW && (warp >> 2) < p.live_chunks) {
        // ---------------- promotion + epilogue: warp = 4 * chunk + lane quarter ----------------
        const int quarter = warp & 3, chunk = warp >> 2;
        const int row = quarter * 32 + lane;                       // weight row inside the tile
        const uint32_t t_lane = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(chunk * CW);
        const float div = 1.0f / (127.0f * 127.0f);

        // activation scales of this CTA's blocks, zero beyond the valid rows: [blocks][BNS] (SRC 1: written by the quantizer;
        // rows beyond M are never stored)
        if (SRC == 0) {
            const int nthreads = live_warps * 32, j0 = k0 * G::BPS;
            const int total = len * G::BPS * BNS;
            for (int i0 = threadIdx.x; i0 < total; i0 += nthreads * 8) {       // eight loads in flight per thread
                float v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int i = i0 + u * nthreads, j = j0 + i / BNS, m = i % BNS;
                    v[u] = (i < total && m < p.M && j < p.nb) ? __ldg(p.sA + (int64_t)j * p.M + m) : 0.0f;
                }
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (i0 + u * nthreads < total) sx[i0 + u * nthreads] = v[u];
            }
            asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory");
        }

        // exchange: CTA `owner` of the cluster finishes this warp's quarter; `slot` is the quarter's place among the owner's
        const int owner = quarter % CL, slot = quarter / CL;
        const int pieces = ((p.M - chunk * CW < CW ? p.M - chunk * CW : CW) + 3) / 4;         // 16-byte pieces per thread that hold live rows
        const uint32_t rx_buf_bytes = rx_bytes(BNS, CL);
        // [owned quarter][chunk][rank of the sender][piece][lane][4 sums]
        auto rx_at = [&](int buf, int from) {
            return base + G::rx_off + (uint32_t)buf * rx_buf_bytes + (uint32_t)((((slot * G::CHUNKS + chunk) * CL + from) * 32 * CW) * 4);
        };

        // Adds one block's terms to the sums, in the reference's order per term: sB * (sA * (float(P) * 1/127^2)), on packed pairs,
        // every operation rounded on its own.  P becomes a float by integer addition onto the bits of 1.5 * 2^23 (|P| < 2^22)
        // and an exact subtraction, which issues four times as fast as the conversion; the sum is written as fma(t, 1, acc), so
        // that the product in front of it cannot be contracted into it.
        uint64_t acc2[CW / 2];
#pragma unroll
        for (int i = 0; i < CW / 2; ++i) acc2[i] = 0ull;
        const uint64_t one2 = pack_f32x2(1.0f, 1.0f), div2 = pack_f32x2(div, div), nmagic2 = pack_f32x2(-kMagic, -kMagic);
        auto add_block = [&](const uint32_t (&v)[CW], float sw, int ks, int blk) {
            if ((k0 + ks) * G::BPS + blk >= p.nb) return;
            const uint32_t sxa = sx_u32 + (uint32_t)(((ks * G::BPS + blk) * BNS + chunk * CW) * 4);
            const uint64_t sw2 = pack_f32x2(sw, sw);
#pragma unroll
            for (int q = 0; q < CW / 4; ++q) {
                uint64_t s[2];
                lds_2xb64(sxa + (uint32_t)(q * 16), s[0], s[1]);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint64_t biased = pack_u32x2(v[q * 4 + 2 * h] + 0x4B400000u, v[q * 4 + 2 * h + 1] + 0x4B400000u);
                    const uint64_t pf = fma_f32x2(biased, one2, nmagic2);                               // float(P), exact
                    acc2[q * 2 + h] = fma_f32x2(f2_mul(sw2, f2_mul(s[h], f2_mul(pf, div2))), one2, acc2[q * 2 + h]);
                }
            }
        };
        auto load_block = [&](uint32_t (&v)[CW], int buf, int blk) {
            const uint32_t ta = t_lane + (uint32_t)(buf * G::ACC_STRIDE + blk * BNS);
            if constexpr (CW == 8) tmem_ld8(ta, v);
            else if constexpr (CW == 16) tmem_ld16(ta, v);
            else tmem_ld32(ta, v);
        };
        auto load_scales = [&](float (&sw)[G::BPS], int stage) {
            const uint32_t sc_u32 = base + (uint32_t)stage * G::STAGE_BYTES + G::W_BYTES + G::X_BYTES + (uint32_t)(row * 4);
#pragma unroll
            for (int blk = 0; blk < G::BPS; ++blk) sw[blk] = lds_f32(sc_u32 + (uint32_t)(blk * kTileRows * 4));
        };
        // A completed accumulator also says that the stage's scales have landed: the MMA issuer had waited for them.
        bool ok = true;
        auto wait_stage = [&](int buf, uint32_t parity) {
            ok = __all_sync(0xffffffffu, mbar_wait(bar(G::ACC_FULL + buf), parity, abort_flag));
            if (!ok && lane == 0) report_timeout(p.status, abort_flag, W_ACC_FULL);
            tc_fence_after();
        };
        auto release_stage = [&](int stage, int buf) {       // accumulators and scales are in registers
            tc_fence_before();
            __syncwarp();
            mbar_arrive_if(bar(G::ACC_EMPTY + buf), lane == 0 ? 1u : 0u);
            mbar_arrive_if(bar(G::EMPTY_AB + stage), lane == 0 ? 1u : 0u);
        };
        // The end of a tile's share: exchange with the cluster and output (`ok` becomes false when a wait has run out).
        auto finish_tile = [&](int r, int tile) {
            float acc[CW];
#pragma unroll
            for (int i = 0; i < CW / 2; ++i) unpack_f32x2(acc2[i], acc[2 * i], acc[2 * i + 1]);
            if (CL > 1) {
                const int rb = p.rx_bufs > 1 ? (r & 1) : 0;
                const uint32_t use = (uint32_t)(p.rx_bufs > 1 ? r >> 1 : r);        // how often this buffer was used before
                const uint32_t full = bar(G::RX_FULL + rb * PW + warp), freed = bar(G::RX_FREE + rb * PW + warp);
                if (owner != rank) {
                    if (!cluster_ready) {
                        cluster_wait();
                        cluster_ready = true;
                    }
                    if (use > 0) ok = __all_sync(0xffffffffu, mbar_wait_cluster(freed, (use - 1) & 1u, abort_flag));
                    if (!ok) {
                        if (lane == 0) report_timeout(p.status, abort_flag, W_PART);
                        return;
                    }
                    const uint32_t to = map_to(rx_at(rb, rank) + (uint32_t)(lane * 16), (uint32_t)owner), to_bar = map_to(full, (uint32_t)owner);
#pragma unroll
                    for (int i = 0; i < CW / 4; ++i)
                        if (i < pieces) send_v4(to + (uint32_t)(i * 512), to_bar, acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]);
                    return;
                }
                if (lane == 0) mbar_expect_tx(full, (uint32_t)((CL - 1) * pieces * 512));
                __syncwarp();
                ok = __all_sync(0xffffffffu, mbar_wait_cluster(full, use & 1u, abort_flag));
                if (!ok) {
                    if (lane == 0) report_timeout(p.status, abort_flag, W_PART);
                    return;
                }
                // parts in ascending K order, this CTA's own (from registers) among them
#pragma unroll
                for (int i = 0; i < CW / 4; ++i) {
                    if (i >= pieces) break;
                    float sum[4];
                    for (int from = 0; from < CL; ++from) {
                        uint32_t w[4] = {__float_as_uint(acc[4 * i]), __float_as_uint(acc[4 * i + 1]), __float_as_uint(acc[4 * i + 2]),
                                         __float_as_uint(acc[4 * i + 3])};
                        if (from != rank) lds_v4(rx_at(rb, from) + (uint32_t)(lane * 16 + i * 512), w[0], w[1], w[2], w[3]);
#pragma unroll
                        for (int u = 0; u < 4; ++u) sum[u] = from == 0 ? __uint_as_float(w[u]) : __fadd_rn(sum[u], __uint_as_float(w[u]));
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) acc[4 * i + u] = sum[u];
                }
                // the buffer may be written again, if it is going to be: the senders wait for this before their next use of it
                if (r + p.rx_bufs < rounds) {
                    if (!cluster_ready) {
                        cluster_wait();
                        cluster_ready = true;
                    }
                    __syncwarp();
                    if (lane < CL && lane != rank) remote_arrive(map_to(freed, (uint32_t)lane));
                    __syncwarp();
                }
            }
            const int n = tile * kTileRows + row;
            if (n < p.N) finish_chunk<CW>(acc, p, chunk * CW, n);
        };

        // one sequence of stages over all tiles of the cluster
        int stage = 0, buf = 0, ks = 0, r = 0, tile = first_tile;
        uint32_t accphase = 0;
        auto next_stage = [&] {
            if (++stage == G::STAGES) stage = 0;
            if (++buf == G::NBUF) { buf = 0; accphase ^= 1u; }
        };
        auto end_of_stage = [&] {
            if (++ks == len) {
                finish_tile(r, tile);
#pragma unroll
                for (int i = 0; i < CW / 2; ++i) acc2[i] = 0ull;
                ks = 0;
                ++r;
                tile += tile_step;
            }
        };
        for (int s = 0; s < my_stages; ++s) {
            wait_stage(buf, accphase);
            if (!ok) break;
            float sw[G::BPS];
            load_scales(sw, stage);
#pragma unroll
            for (int b0 = 0; b0 < G::BPS; b0 += G::VB) {
                uint32_t v[G::VB][CW];
#pragma unroll
                for (int q = 0; q < G::VB; ++q) load_block(v[q], buf, b0 + q);
                tmem_wait_ld();
                if (b0 + G::VB == G::BPS) release_stage(stage, buf);
#pragma unroll
                for (int q = 0; q < G::VB; ++q) add_block(v[q], sw[b0 + q], ks, b0 + q);
            }
            next_stage();
            end_of_stage();
            if (!ok) break;
        }
    }

    // ---------------- teardown ----------------
    tc_fence_before();
    __syncthreads();
    const bool gave_up = lds_volatile_u32(abort_flag) != 0u;
    if (warp == MW) {
        tc_fence_after();
        tmem_dealloc(tmem_base, G::TMEM_COLS);
    }
    // No CTA leaves while another of its cluster may still write into its shared memory.
    __syncwarp();
    if (!cluster_ready) cluster_wait();
    cluster_arrive();
    cluster_wait();
    // A CTA that gave up has not waited for everything that was sent to it, and the barrier orders the sending of an asynchronous
    // store, not its arrival: it stays for 0.2 ms, where such a store takes a microsecond.
    if (gave_up) {
        const long long t0 = clock64();
        while (clock64() - t0 < 400000ll) __nanosleep(1000);
    }
}

// Row-wise block quantizer for the few activation rows of a decode step (same arithmetic as the standalone quantizer:
// quant_math.cuh), used by the quantize-on-load entry point in front of the GEMM.  A thread takes 8 consecutive elements;
// the QB/8 lanes of a block reduce the absmax with xor shuffles.  It lets the GEMM, launched with programmatic stream
// serialisation, become resident at once: the GEMM's set-up and its first weight copies run beside this kernel and
// only its activation loads wait for it.
template <int QB>
__global__ void __launch_bounds__(256) skinny_quantize_kernel(const void* __restrict__ x, int x_dtype, int64_t ldx,
                                                              int8_t* __restrict__ q, float* __restrict__ sx, int M, int K, int nb) {
    // Launched with programmatic stream serialisation itself: resident while the kernel before it (the previous layer's
    // reduction) finishes.  Its own dependent, the GEMM, is released only after that kernel has completed, so that
    // whatever the GEMM reads early (weights, weight scales) has been at rest for a full kernel boundary.
    after_predecessor();
    constexpr int LPB = QB / 8;
    const int upr = nb * LPB;                                  // units per row, padded to whole blocks
    const int64_t u = (int64_t)blockIdx.x * 256 + threadIdx.x;
    const int m = (int)(u / upr), piece = (int)(u % upr), k = piece * 8;
    const bool wide = x_dtype == BI8_F32;
    const bool valid = m < M && k < K;
    float f[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = 0.0f;
    if (valid) {
        const unsigned char* src = static_cast<const unsigned char*>(x) + ((int64_t)m * ldx + k) * (wide ? 4 : 2);
        const uint4 a = ld_nc_v4(src);
        if (wide) {
            const uint4 b = ld_nc_v4(src + 16);
            f[0] = __uint_as_float(a.x); f[1] = __uint_as_float(a.y); f[2] = __uint_as_float(a.z); f[3] = __uint_as_float(a.w);
            f[4] = __uint_as_float(b.x); f[5] = __uint_as_float(b.y); f[6] = __uint_as_float(b.z); f[7] = __uint_as_float(b.w);
        } else {
            const uint32_t w4[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                if (x_dtype == BI8_BF16) {
                    f[2 * h] = bf16lo(w4[h]);
                    f[2 * h + 1] = bf16hi(w4[h]);
                } else {
                    const float2 t2 = __half22float2(*reinterpret_cast<const __half2*>(&w4[h]));
                    f[2 * h] = t2.x;
                    f[2 * h + 1] = t2.y;
                }
            }
        }
    }
    float amax = 0.0f;
#pragma unroll
    for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(f[e]));
#pragma unroll
    for (int off = 1; off < LPB; off <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    if (!valid) return;
    BlockQ bq;
    bq.set(amax, !wide);
    const uint32_t lo = pack4(bq.q(f[0]), bq.q(f[1]), bq.q(f[2]), bq.q(f[3]));
    const uint32_t hi = pack4(bq.q(f[4]), bq.q(f[5]), bq.q(f[6]), bq.q(f[7]));
    *reinterpret_cast<uint2*>(q + (int64_t)m * K + k) = make_uint2(lo, hi);
    if ((piece % LPB) == 0) sx[(int64_t)(k / QB) * M + m] = amax;
}

// Row-parallel layer: the GEMM has left this rank's partial result in `part` (fp32 [M, N]); this kernel exchanges it with the
// other ranks over peer memory (peer_common.cuh) and writes the layer's output.  A thread takes four consecutive columns.
// Launched as a programmatic dependent of the GEMM: resident while it runs.
__global__ void __launch_bounds__(kPeerThreads) skinny_reduce_peer_kernel(const float* __restrict__ part, int M, int N, const PeerArgs a,
                                                                          const void* bias, int bias_dtype, void* out, int out_dtype,
                                                                          long long limit_cycles, int* status) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int64_t count = (int64_t)M * N;
    const int64_t i = (int64_t)blockIdx.x * kPeerChunk + (int64_t)threadIdx.x * 4;
    const uint32_t seq = peer_sequence(a);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < count) v = __ldcg(reinterpret_cast<const float4*>(part + i));
    peer_exchange_store(a, seq, v, count, N, bias, bias_dtype, out, out_dtype, limit_cycles, status);
}

template <int QB_, int BNS_, int SRC_>
struct Instance {
    static constexpr int QB = QB_, BNS = BNS_, SRC = SRC_;
};

// ---- host ---------------------------------------------------------------------------------------------------------------
// How many clusters of a size fit on the device at once (one CTA per SM): asked once per device, for one kernel of the family.
struct ClusterSlots {
    int n[kMostCluster + 1] = {0};
    bool known = false;
};

template <int QB, int BNS, int SRC>
int launch_skinny(const GemmArgs& g, const SkParams& p, int cluster, int clusters, size_t smem, cudaStream_t st) {
    using G = SkGeo<QB, BNS, SRC>;
    CUtensorMap mw, mx, ms;
    int dev = 0;
    BI8_CUDA_TRY(current_device(&dev));
    int rc = cached_operand_map(&mw, dev, g.Bt, g.N, g.K, g.ldb, kTileRows);
    if (rc != BI8_OK) return rc;
    mx = mw;                        // SRC 1: not used, the kernel writes the activation tiles itself
    if (SRC == 0) {
        rc = cached_operand_map(&mx, dev, g.A, g.M, g.K, g.lda, BNS);
        if (rc != BI8_OK) return rc;
    }
    rc = cached_scale_map(&ms, dev, g.sB, p.nb, g.N, kTileRows, G::BPS);
    if (rc != BI8_OK) return rc;
    static SmemOptIn opt_in;
    rc = opt_in.ensure(gemm_tc_skinny_kernel<QB, BNS, SRC>, smem);
    if (rc != BI8_OK) return rc;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(cluster * clusters));
    cfg.blockDim = dim3(G::THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;    // what may run before the predecessor has completed: early_weights
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    BI8_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_tc_skinny_kernel<QB, BNS, SRC>, mw, mx, ms, p));
    return BI8_OK;
}

constexpr size_t kSmemLimit = 227 * 1024;

int cluster_slots(ClusterSlots* out, int sms) {
    static ClusterSlots table[64];
    static std::mutex mu;
    int dev = 0;
    BI8_CUDA_TRY(current_device(&dev));
    if (dev < 0 || dev >= 64) return fail(BI8_ERR_CUDA, "device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lock(mu);
    ClusterSlots& t = table[dev];
    if (!t.known) {
        BI8_CUDA_TRY(cudaFuncSetAttribute(gemm_tc_skinny_kernel<64, 64, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit));
        t.n[1] = sms;
        for (int c = 2; c <= kMostCluster; c *= 2) {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3((unsigned)(c * (sms / c)));
            cfg.blockDim = dim3(SkGeo<64, 64, 0>::THREADS);
            cfg.dynamicSmemBytes = kSmemLimit;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = (unsigned)c;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            BI8_CUDA_TRY(cudaOccupancyMaxActiveClusters(&t.n[c], gemm_tc_skinny_kernel<64, 64, 0>, &cfg));
        }
        t.known = true;
    }
    *out = t;
    return BI8_OK;
}

int bns_for(int64_t M) { return M <= 16 ? 16 : M <= 32 ? 32 : 64; }
int64_t stages_of(int64_t K, int bns) {
    const int64_t ks = bns == 16 ? SkGeo<64, 16, 0>::KS : bns == 32 ? SkGeo<64, 32, 0>::KS : SkGeo<64, 64, 0>::KS;
    return (K + ks - 1) / ks;
}

// f(Instance<...>) for the kernel instance of (block, bns, src), or `otherwise` where none is built.  The dispatcher quantizes inside the
// kernel up to 16 rows; the instances with 32 serve callers that ask for it or have no scratch (BI8_GEMM_QUANT_IN_KERNEL).
template <typename R, typename F>
R with_instance(int block, int bns, int src, R otherwise, F f) {
#define BI8_SK(QB, BNS)                                          \
    if (block == QB && bns == BNS) {                             \
        if (src == 0) return f(Instance<QB, BNS, 0>{});          \
        if constexpr (BNS <= 32) return f(Instance<QB, BNS, 1>{}); \
    }
    BI8_SK(32, 16) BI8_SK(32, 32) BI8_SK(32, 64)
    BI8_SK(64, 16) BI8_SK(64, 32) BI8_SK(64, 64)
    BI8_SK(128, 16) BI8_SK(128, 32) BI8_SK(128, 64)
#undef BI8_SK
    return otherwise;
}

// The cluster size: the one with the fewest stages from the first to the last.  The exchange of partial sums, and with it the
// wait for the slowest of the cluster, counts as kExchange stages (measured at 8, 32 and 64 rows over ten layer shapes: 1.5,
// 2.5 and 5.5 us for 2, 4 and 8 CTAs where a stage takes 0.4 us).  It depends on the shape alone (not on where the activations come
// from), because it decides how the sums associate.
struct SkPlan {
    int cluster = 1, clusters = 1;
    int64_t cost = 0;                       // in stages
};
constexpr int kExchange[3][kMostCluster + 1] = {{0, 0, 4, 0, 6, 0, 0, 0, 14}, {0, 0, 2, 0, 4, 0, 0, 0, 8}, {0, 0, 3, 0, 7, 0, 0, 0, 14}};
int split_plan(int64_t N, int64_t K, int block, int bns, int sms, SkPlan* pl) {
    ClusterSlots slots;
    const int rc = cluster_slots(&slots, sms);
    if (rc != BI8_OK) return rc;
    const int64_t tiles = (N + kTileRows - 1) / kTileRows, nks = stages_of(K, bns);
    int64_t best = -1;
    // sizes at which the activations' operand tiles fit as well (SRC 1), else those at which the ring does
    for (int src = bns == 16 ? 1 : 0; src >= 0 && best < 0; --src) {
        for (int c = 1; c <= kMostCluster && c <= nks; c *= 2) {
            const int fit = slots.n[c];
            if (fit < 1) continue;
            const size_t smem = with_instance(block, bns, src, (size_t)0, [&](auto in) {
                using I = decltype(in);
                return smem_of<I::QB, I::BNS, I::SRC>((int)((nks + c - 1) / c), c, tiles > fit ? 2 : 1);
            });
            if (smem == 0 || smem > kSmemLimit) continue;
            const int64_t cost = (tiles + fit - 1) / fit * ((nks + c - 1) / c) + kExchange[bns == 16 ? 0 : bns == 32 ? 1 : 2][c];
            if (best < 0 || cost < best) {
                best = pl->cost = cost;
                pl->cluster = c;
                pl->clusters = (int)(tiles < fit ? tiles : fit);
            }
        }
    }
    if (best < 0) pl->cluster = 0;          // no size fits
    return BI8_OK;
}

// What a launch needs beside the operands; `smem` 0: no kernel instance, or it does not fit.
struct SkLaunch {
    SkPlan plan;
    int share = 0, rx_bufs = 1;
    uint32_t sx_off = 0, xq_off = 0;
    size_t smem = 0;
};
int plan_launch(const GemmArgs& g, int sms, SkLaunch* out) {
    const int rc = split_plan(g.N, g.K, g.block, bns_for(g.M), sms, &out->plan);
    if (rc != BI8_OK || out->plan.cluster == 0) return rc;
    const int64_t tiles = (g.N + kTileRows - 1) / kTileRows, nks = stages_of(g.K, bns_for(g.M));
    const int c = out->plan.cluster;
    out->share = (int)((nks + c - 1) / c);
    out->rx_bufs = tiles > out->plan.clusters ? 2 : 1;
    out->smem = with_instance(g.block, bns_for(g.M), g.X != nullptr ? 1 : 0, (size_t)0, [&](auto in) {
        using I = decltype(in);
        return smem_of<I::QB, I::BNS, I::SRC>(out->share, c, out->rx_bufs, &out->sx_off, &out->xq_off);
    });
    if (out->smem > kSmemLimit) out->smem = 0;
    return BI8_OK;
}

// conditions that depend on the shape only
bool skinny_shape_ok(int64_t M, int64_t N, int64_t K, int block) {
    if (M < 1 || M > kSkMaxM || N < 1 || K < 1) return false;
    if (block != 32 && block != 64 && block != 128) return false;
    return N % 4 == 0 && N < (1ll << 30) && K < (1ll << 30);
}

}  // namespace

int launch_skinny_quantize(const void* x, int x_dtype, int64_t ldx, int8_t* q, float* sx, int64_t M, int64_t K, int block,
                           cudaStream_t st) {
    const int nb = (int)((K + block - 1) / block);
    const int64_t units = M * nb * (block / 8);
    const unsigned blocks = (unsigned)((units + 255) / 256);
    switch (block) {
        case 32: return launch_chained(skinny_quantize_kernel<32>, blocks, 256, 0, st, x, x_dtype, ldx, q, sx, (int)M, (int)K, nb);
        case 64: return launch_chained(skinny_quantize_kernel<64>, blocks, 256, 0, st, x, x_dtype, ldx, q, sx, (int)M, (int)K, nb);
        case 128: return launch_chained(skinny_quantize_kernel<128>, blocks, 256, 0, st, x, x_dtype, ldx, q, sx, (int)M, (int)K, nb);
        default: return fail(BI8_ERR_BLOCK, "skinny quantizer supports block 32, 64, 128 (got %d)", block);
    }
}

bool gemm_skinny_applicable(const GemmArgs& g) {
    if (g.partials != nullptr || !skinny_shape_ok(g.M, g.N, g.K, g.block)) return false;
    const DeviceInfo di = device_info();
    if (!di.ok) return false;
    if (!aligned(g.Bt, 16) || g.ldb % 16 != 0 || !aligned(g.sB, 16)) return false;
    if (g.X != nullptr) {
        // quantization inside the kernel reads 8 elements (16 or 32 bytes) at a time
        const int esz = g.x_dtype == BI8_F32 ? 4 : 2;
        if (g.M > 32 || !aligned(g.X, 16) || (g.ldx * esz) % 16 != 0 || g.K % 8 != 0 || (g.X2 != nullptr && !aligned(g.X2, 16))) return false;
    } else if (!aligned(g.A, 16) || g.lda % 16 != 0) {
        return false;
    }
    SkLaunch l;
    return plan_launch(g, di.sms, &l) == BI8_OK && l.smem != 0;
}

// Activation values that a CTA quantizes where the kernel does it itself.
int64_t gemm_skinny_part(const GemmArgs& g) {
    SkLaunch l;
    if (!skinny_shape_ok(g.M, g.N, g.K, g.block) || plan_launch(g, device_info().sms, &l) != BI8_OK || l.plan.cluster == 0) return INT64_MAX;
    return g.M * ((g.K + l.plan.cluster - 1) / l.plan.cluster);
}

// Whether this kernel is taken.  Up to 32 rows it always is.  From 33 on its promotion costs as much as the weights take to arrive, and the
// general kernel, whose terms are rounded differently, overtakes it where it fills the SMs: it is taken where a model says that
// it gains 2.5 us (estimates in microseconds, the time of a stage by the blocks it promotes).  The present general kernel is faster than
// that model: at 64 rows, general against here, block 32 / 64 / 128: taken there 4096 x 11008 31.8, 42.8 / 20.9, 31.7 / 16.7, 26.4; 5120 x
// 5120 22.3, 30.3 / 15.1, 20.3 / 12.5, 16.0; kept here 8192 x 8192 55.4, 46.7 / 32.5, 30.7 / 23.8, 23.9; 11008 x 4096 34.8, 34.3 / (taken) 21.8,
// 23.6 / 16.7, 18.9; 4096 x 4096 17.9, 17.6 / 12.8, 13.7 / 11.0, 12.1; 1024 x 1024 6.9, 10.0 / 6.2, 8.3 / 6.5, 7.6; 2048 x 2048 at 64 8.8, 11.3.
// In 48 shapes of 33, 40 and 64 rows the general kernel is nowhere taken and more than 3 % slower; in a third this one is kept and 5 % or more
// slower, by 3.1 us at most.  The line does not follow the general kernel's speed, because its error is the larger one: against 64
// bits, fp32 results, 1.1-1.5e-7 where this kernel has 0.5-1.2e-7 (K up to 4096; 11008: 1.4-1.9e-7 and 1.0-1.8e-7).
bool gemm_skinny_preferred(const GemmArgs& g) {
    if (!gemm_skinny_applicable(g)) return false;
    if (g.M <= 32) return true;
    SkLaunch l;
    const char* why = "";
    if (plan_launch(g, device_info().sms, &l) != BI8_OK || !gemm_tc_applicable(g, &why)) return true;
    const double stage_us = g.block <= 32 ? 1.2 : g.block <= 64 ? 0.9 : 0.7;
    return stage_us * (double)l.plan.cost + 2.0 <= gemm_tc_estimate_us(g) + 2.5;
}

int launch_gemm_skinny(const GemmArgs& g, cudaStream_t st) {
    const DeviceInfo di = device_info();
    if (!di.ok) return fail(BI8_ERR_CUDA, "tensor-core GEMM needs a compute capability 10.x device");
    SkLaunch l;
    int rc = plan_launch(g, di.sms, &l);
    if (rc != BI8_OK) return rc;
    if (l.smem == 0) return fail(BI8_ERR_SHAPE, "skinny tensor-core GEMM: the shape's shared memory does not fit");
    SkParams p;
    std::memset(&p, 0, sizeof(p));
    p.sA = g.sA;
    p.X = g.X;
    p.X2 = g.X2;
    p.ldx = g.ldx;
    p.eps = g.eps;
    p.op = g.pre_op;
    p.x_dtype = g.x_dtype;
    p.bias = g.bias;
    p.bias_ld = g.bias_ld;
    p.C = g.C;
    p.status = device_status_ptr();
    if (!p.status) return BI8_ERR_CUDA;
    p.ldc = g.ldc;
    p.M = (int)g.M;
    p.N = (int)g.N;
    p.K = (int)g.K;
    p.nb = (int)((g.K + g.block - 1) / g.block);
    p.nks = (int)stages_of(g.K, bns_for(g.M));
    p.tiles = (int)((g.N + kTileRows - 1) / kTileRows);
    p.out_dtype = g.out_dtype;
    p.bias_dtype = g.bias_dtype;
    const int bns = bns_for(g.M), cw = bns / 2;
    p.live_chunks = (int)((g.M + cw - 1) / cw);
    p.early_weights = g.after_own_quantizer ? 1 : 0;
    p.rx_bufs = l.rx_bufs;
    p.share = l.share;
    p.sx_off = l.sx_off;
    p.xq_off = l.xq_off;
    rc = with_instance(g.block, bns, g.X != nullptr ? 1 : 0, (int)BI8_ERR_SHAPE, [&](auto in) {
        using I = decltype(in);
        return launch_skinny<I::QB, I::BNS, I::SRC>(g, p, l.plan.cluster, l.plan.clusters, l.smem, st);
    });
    if (rc != BI8_OK || g.peer == nullptr) return rc;
    // row-parallel layer: a kernel behind this one exchanges the partial results with the other ranks and writes the layer's output
    const PeerEpilogue& pe = *g.peer;
    const int64_t count = g.M * g.N;
    return launch_chained(skinny_reduce_peer_kernel, (unsigned)((count + kPeerChunk - 1) / kPeerChunk), kPeerThreads, 0, st, (const float*)g.C,
                          (int)g.M, (int)g.N, *static_cast<const PeerArgs*>(pe.args), pe.bias, pe.bias_dtype, pe.out, pe.out_dtype, pe.limit_cycles,
                          p.status);
}

}  // namespace bi8
