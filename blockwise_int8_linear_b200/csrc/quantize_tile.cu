// Tile quantizer: column-wise (fused transpose) quantize, and the dual quantizer that also produces the row-wise
// result from the same read of the input.
//
// Semantics (paths inside the reference project):
//   column-wise  block_linear.py:93-94, 100-103   x.t().contiguous() followed by the row-wise quantizer
//   row-wise     triton_functions.py:382-406      scale = max|x| over the block, q = rint(127 * (x / scale))
// Both results are bit-identical to the single-purpose kernels of quantize.cu (same BlockQ arithmetic).
//
// Persistent CTAs walk over tiles of 128 rows x 128 columns of a 16-bit input:
//   * one elected thread fetches the tile with two TMA loads (64 columns = 128 bytes wide each, 128-byte swizzle) that
//     complete on an mbarrier; rows and columns outside the tensor arrive as zeros.
//   * Inputs whose rows are not 16-byte aligned, which a tensor map cannot describe (a 50257-wide vocabulary): rows eight
//     apart share an alignment, so a tensor map whose "rows" are eight rows long describes them.  Eight TMA loads (kOct) fetch
//     the 16 rows of a tile that are equal modulo 8, 136 columns from the 16-byte boundary at or before the tile's first.
//     The threads shift what they read by the class's offset, which is a constant for the column-wise role's unrolled
//     rows and, with a warp per class, for a whole warp of the row-wise role.  8192 x 50257: dual 494 -> 399 us (345 with aligned
//     rows), column-wise 488 -> 224 (225); with one operation per pair (quant_math.cuh) dual 338 (288), and 8192 x 8192, aligned, 63.5 -> 54.4,
//     8192 x 3072 30.8 -> 26.6.  What is left is the rest of the instructions: with twice the threads and half the words for each (64 registers, no
//     spills) every one of those times was a tenth longer.
//     Where the number of rows is not a multiple of 8 (kShift) all threads fetch: a half-warp reads a tile row as aligned
//     16-byte pieces, shifts the bytes into place between neighbouring lanes and stores them where the TMA would have put
//     them.  The loads of the next tile are in flight, in registers, while the current one is quantized.  (A zero-padded
//     copy in front of the kernel cost one more pass: 0.9 ms for a 8192 x 50257 matrix.)
//   * column-wise: a thread owns a pair of adjacent columns and 32 rows.  It reads them as 32 four-byte words (all lanes
//     of a warp read one row: conflict free under the swizzle), takes the absmax of both columns with packed 16-bit
//     max instructions, exchanges it with the other row groups of its block through shared memory, and quantizes
//     both columns at once with packed fp32 arithmetic.  The bytes go into a transposed tile [column][row];
//   * row-wise (dual only): a thread owns 64 consecutive columns of one row (16-byte loads, eight rows per
//     quarter-warp: conflict free under the swizzle) and writes 64 bytes into a row-major tile;
//   * SUM (dual): the column-wise role has every value in a register when it quantizes, so the column sums of the tile (the bias
//     gradient, out of a gradient) cost its 32 additions per column and no read of their own: 8192 x 768 x 3072 forward and
//     backward 226 -> 213 us.  fp32, rows ascending, one partial row per tile; column_sum.cu adds those.  Where the threads fetch
//     the input themselves (kShift) the sums of fp16 spill a few registers, and still cost less than a read of their own: with sums / with a separate
//     column sum / without, block 64: 8190 x 3071 bf16 48 / 71 / 44 us, fp16 56 / 75 / 48, 8190 x 50257 472 / 716 / 466 and 601 / 759 / 509.
//   * the two int8 tiles leave with one TMA store each (128-byte swizzle again, so that the transposed writes do not
//     pile up on a few banks); tile parts outside the tensors are clipped by the store.
// The input tile has three stages (two in the column-wise kernel), so the next loads are in flight while a tile is quantized;
// in the dual kernel the two quantizations run side by side in two groups of 256 threads (one CTA of 512 threads per SM;
// the column-wise kernel alone runs two CTAs of 256).
#include "bi8_common.cuh"
#include "quant_math.cuh"
#include "tc_common.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

namespace bi8 {
namespace {

using namespace ptx;

constexpr int kQT = 128;          // tile edge (rows and columns)
constexpr int kQThreads = 256;
enum { QW_LOAD = 1, QW_EMPTY = 2 };

// shared memory layout (offsets from a 1024-byte aligned base) for NST input stages
enum InputKind { kTiled = 0, kShift = 1, kOct = 2 };   // how a tile is fetched
constexpr uint32_t kInStage = 2 * kQT * 128;          // two sub-tiles [128 rows][128 bytes]
constexpr int kOctCols = kQT + 8;                     // kOct: columns fetched
constexpr uint32_t kOctRow = kOctCols * 2, kOctClass = kQT / 8 * kOctRow, kOctStage = 8 * kOctClass;   // [8 classes][16 rows][272 bytes]
static_assert(kOctClass % 128 == 0 && kOctStage % 1024 == 0, "TMA destinations");
template <int NST, int IN>
struct QLayout {
    static constexpr uint32_t in_off = 0, in_stage = IN == kOct ? kOctStage : kInStage;
    static constexpr uint32_t outc_off = NST * in_stage;              // [128 columns][128 row bytes]
    static constexpr uint32_t ex_off = outc_off + kQT * 128;          // absmax exchange [4 row groups][128 columns] fp32
    static constexpr uint32_t sum_off = ex_off + 4 * kQT * 4;         // column sums of the row groups (dual only)
    static constexpr uint32_t bar_off = sum_off + 4 * kQT * 4;        // 2 * NST barriers and the abort flag
    static constexpr uint32_t outr_off = bar_off + 1024;              // [128 rows][128 column bytes]   (dual only)
    static constexpr uint32_t bytes_col = outr_off, bytes_dual = outr_off + kQT * 128;
    static_assert(outr_off % 1024 == 0 && outc_off % 1024 == 0, "swizzled tiles start on 1024-byte boundaries");
};

// byte offset of 16-byte chunk `chunk` of row `row` in a [rows][128 bytes] tile written or read by TMA with the 128-byte swizzle
__device__ __forceinline__ uint32_t swz(int row, int chunk) { return (uint32_t)(row * 128 + ((chunk ^ (row & 7)) << 4)); }

template <typename T>
struct Pk;
template <>
struct Pk<__nv_bfloat16> {
    // max(|a|, m) on both 16-bit halves; a NaN operand is ignored, like fmaxf
    static __device__ __forceinline__ uint32_t absmax(uint32_t a, uint32_t m) {
        __nv_bfloat162 r = __hmax2(__habs2(*reinterpret_cast<__nv_bfloat162*>(&a)), *reinterpret_cast<__nv_bfloat162*>(&m));
        return *reinterpret_cast<uint32_t*>(&r);
    }
    static __device__ __forceinline__ void unpack(uint32_t w, float& lo, float& hi) {
        lo = bf16lo(w);
        hi = bf16hi(w);
    }
};
template <>
struct Pk<__half> {
    static __device__ __forceinline__ uint32_t absmax(uint32_t a, uint32_t m) {
        __half2 r = __hmax2(__habs2(*reinterpret_cast<__half2*>(&a)), *reinterpret_cast<__half2*>(&m));
        return *reinterpret_cast<uint32_t*>(&r);
    }
    static __device__ __forceinline__ void unpack(uint32_t w, float& lo, float& hi) {
        float2 f = __half22float2(*reinterpret_cast<__half2*>(&w));
        lo = f.x;
        hi = f.y;
    }
};

// Quantizer of a pair of values with (possibly different) block scales, on packed fp32 pairs.  The same operations, in
// the same order and each rounded on its own, as BlockQ::q: kOnce fma(x, r127, magic); kFast q0 = x*r, e = fma(-s, q0, x), y = fma(e, r, q0),
// z = 127*y, z + magic (written as fma(z, 1, magic) so that the multiply cannot be contracted into the addition).
enum QuantWay { kOnce = 0, kFast = 1, kDivide = 2 };
struct PairQ {
    BlockQ lo, hi;
    uint64_t r2, ns2;             // kFast; packed in its loop they cost fp16 up to 12 bytes of spills more
    bool fast, once;
    __device__ __forceinline__ void set(float amax_lo, float amax_hi) {
        lo.set(amax_lo, true);
        hi.set(amax_hi, true);
        fast = lo.fast && hi.fast;
        once = lo.once && hi.once;
        r2 = f2_pack(lo.rcp, hi.rcp);
        ns2 = f2_pack(-amax_lo, -amax_hi);
    }
    // The way is chosen by the caller around its whole loop (choose) rather than per pair.
    template <int WAY>
    __device__ __forceinline__ void q(float xlo, float xhi, uint32_t& blo, uint32_t& bhi) const {
        if (WAY == kOnce) {
            f2_bits(f2_fma(f2_pack(xlo, xhi), f2_pack(lo.r127(), hi.r127()), f2_pack(kMagic, kMagic)), blo, bhi);
        } else if (WAY == kFast) {
            const uint64_t c127 = f2_pack(127.0f, 127.0f), cmagic = f2_pack(kMagic, kMagic), cone = f2_pack(1.0f, 1.0f);
            const uint64_t v2 = f2_pack(xlo, xhi);
            const uint64_t q0 = f2_mul(v2, r2);
            const uint64_t e = f2_fma(ns2, q0, v2);
            const uint64_t y = f2_fma(e, r2, q0);
            f2_bits(f2_fma(f2_mul(c127, y), cone, cmagic), blo, bhi);
        } else {
            blo = lo.q(xlo);
            bhi = hi.q(xhi);
        }
    }
    // f(the way of this thread's pairs).  bf16: one operation or the division; `once` is `fast` there, and it is `fast` that is asked, because that is what
    // keeps the five operations out of the division's code (of zero blocks, rows behind the last, a last tile of few columns).  fp16: with ONCE one operation where that
    // holds for the whole warp, because a warp that is divided would do both; the third way's code costs registers, which kShift does not
    // have (dual, 8190 x 3071: 49 us without, 56 with) and kOct and the column-wise kernel gain nothing from (26.6, 28.7; dual tiles 30.7, 28.7).
    // FIVE: bf16 by the five operations (see five_operations).
    template <typename T, bool ONCE, bool FIVE, typename F>
    __device__ __forceinline__ void choose(F f) const {
        if constexpr (std::is_same_v<T, __nv_bfloat16> && !FIVE) {
            if (fast) f(std::integral_constant<int, kOnce>{});
            else f(std::integral_constant<int, kDivide>{});
        } else {
            if (ONCE && __all_sync(0xffffffffu, once)) f(std::integral_constant<int, kOnce>{});
            else if (fast) f(std::integral_constant<int, kFast>{});
            else f(std::integral_constant<int, kDivide>{});
        }
    }
};

// Barrier among the `n` threads of one role (named barrier `id`) that also tells every one of them whether all of them
// came with `ok` set: a wait that ran out in some thread ends the loop in all threads of the role, so that no thread is
// left waiting at a barrier the others will never reach.
__device__ __forceinline__ bool role_barrier_all(int id, int n, bool ok) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"(ok ? 1u : 0u), "r"(id), "r"(n)
        : "memory");
    return r != 0u;
}
__device__ __forceinline__ void role_barrier(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }

// Persistent CTAs walk over the tiles; the input tile has two or three stages (full / empty mbarriers per stage, the
// loads of the next tiles are in flight while the current one is quantized, and a stage is released as soon as every thread
// has its part of it in registers).  256 threads do the column-wise work; in the dual kernel 256 more do the row-wise work on the
// same tile at the same time.  Each role has its own named barrier and its own elected thread for the TMA store of its
// output tile, so neither waits for the other.
// One tile of an input with unaligned rows, by NT threads: a half-warp has the 16 16-byte chunks of a row, the two half-warps have
// rows r and r + 8, whose byte offset from a 16-byte boundary is the same (the row pitch is even), so that the shift is the
// same in all lanes of a warp.  Per step, warp w of NT / 32 takes the row pairs w, w + NT / 32, ...
template <int NT>
struct ShiftLoader {
    static constexpr int STEPS = kQT * 16 / NT;
    uint4 piece[STEPS];           // the aligned 16 bytes at or before the chunk's first byte
    uint4 last[STEPS];            // lane 15 of a half-warp: the 16 bytes behind its own
    const unsigned char* x;
    int64_t pitch;                // bytes
    int R, C;

    static __device__ __forceinline__ int tile_row(int tid, int step) {
        const int g = (tid >> 5) + step * (NT / 32);
        return (g >> 3) * 16 + (g & 7) + 8 * ((tid >> 4) & 1);
    }
    // Requests the pieces of the tile at (r0, c0).  A piece is read only where it contains a byte of the row's part inside the
    // tile, so no access leaves the tensor's 16-byte granules.
    __device__ __forceinline__ void request(int tid, int r0, int c0) {
        const int i = tid & 15;
        const unsigned char* tile = x + (int64_t)r0 * pitch + (int64_t)c0 * 2;
        if (r0 + kQT <= R && c0 + kQT <= C) {
#pragma unroll
            for (int u = 0; u < STEPS; ++u) {
                const uintptr_t a = reinterpret_cast<uintptr_t>(tile + (int64_t)tile_row(tid, u) * pitch);
                const void* at = reinterpret_cast<const void*>((a & ~(uintptr_t)15) + 16 * i);
                piece[u] = ld_nc_v4(at);
                if (i == 15 && (a & 15u) != 0) last[u] = ld_nc_v4(static_cast<const unsigned char*>(at) + 16);
            }
        } else {
            const int cols = C - c0 < kQT ? C - c0 : kQT;
#pragma unroll
            for (int u = 0; u < STEPS; ++u) {
                piece[u] = last[u] = make_uint4(0u, 0u, 0u, 0u);
                if (r0 + tile_row(tid, u) < R) {
                    const uintptr_t a = reinterpret_cast<uintptr_t>(tile + (int64_t)tile_row(tid, u) * pitch);
                    const uintptr_t end = a + (uintptr_t)cols * 2, at = (a & ~(uintptr_t)15) + 16 * i;
                    if (at < end) piece[u] = ld_nc_v4(reinterpret_cast<const void*>(at));
                    if (i == 15 && (a & 15u) != 0 && at + 16 < end) last[u] = ld_nc_v4(reinterpret_cast<const void*>(at + 16));
                }
            }
        }
    }
    // Shifts the requested bytes into place and stores the tile at shared address `tile` (two swizzled 128 x 128-byte halves);
    // elements outside the tensor become zero.  All lanes of a warp call it together.
    __device__ __forceinline__ void store(int tid, int r0, int c0, uint32_t tile) {
        const int i = tid & 15;
        const bool edge = r0 + kQT > R || c0 + kQT > C;
        const uint32_t dst = tile + (uint32_t)((i >> 3) * kQT * 128);
        const uint32_t base_off = (uint32_t)(reinterpret_cast<uintptr_t>(x) + (uintptr_t)c0 * 2), p32 = (uint32_t)pitch;
#pragma unroll
        for (int u = 0; u < STEPS; ++u) {
            const int tr = tile_row(tid, u);
            const uint32_t off = (base_off + (uint32_t)(r0 + tr) * p32) & 15u, bits = (off & 2u) * 8u;
            const uint32_t own[4] = {piece[u].x, piece[u].y, piece[u].z, piece[u].w};
            const uint32_t tail[4] = {last[u].x, last[u].y, last[u].z, last[u].w};
            uint32_t w[4];
            auto shifted = [&](auto words) {              // the row's bytes begin `WS` words (and `bits` bits) into the piece
                constexpr int WS = decltype(words)::value;
                uint32_t r[5];
#pragma unroll
                for (int k = 0; k < 5; ++k) {
                    if (k + WS < 4) {
                        r[k] = own[(k + WS) & 3];
                    } else {
                        const uint32_t next = __shfl_down_sync(0xffffffffu, own[(k + WS) & 3], 1);
                        r[k] = i == 15 ? tail[(k + WS) & 3] : next;
                    }
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) w[k] = __funnelshift_r(r[k], r[k + 1], bits);
            };
            if (off < 4u) shifted(std::integral_constant<int, 0>{});
            else if (off < 8u) shifted(std::integral_constant<int, 1>{});
            else if (off < 12u) shifted(std::integral_constant<int, 2>{});
            else shifted(std::integral_constant<int, 3>{});
            if (edge) {
                const int valid = r0 + tr < R ? C - (c0 + 8 * i) : 0;          // elements of the chunk inside the tensor
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (2 * k >= valid) w[k] = 0u;
                    else if (2 * k + 1 >= valid) w[k] &= 0xffffu;
                }
            }
            sts_v4(dst + swz(tr, i & 7), w[0], w[1], w[2], w[3]);
        }
    }
};

template <typename T, int B, bool DUAL, int IN, bool SUM, bool FIVE>
__global__ void __launch_bounds__(DUAL ? 2 * kQThreads : kQThreads, DUAL ? 1 : 2)
quantize_tile_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmQc,
                     const __grid_constant__ CUtensorMap tmQr, const void* __restrict__ x, int64_t ldx, float* __restrict__ s_col,
                     float* __restrict__ s_row, float* __restrict__ sums, int R, int C, int col_tiles, int num_tiles, int* status) {
    static_assert(B == 32 || B == 64 || B == 128, "block sizes of the tile quantizer");
    constexpr int NT = DUAL ? 2 * kQThreads : kQThreads;
    constexpr int NST = DUAL ? 3 : 2;                      // input stages: the loads of the next NST - 1 tiles are in flight
    using L = QLayout<NST, IN>;
    constexpr bool SHIFT = IN == kShift, OCT = IN == kOct;
    constexpr long long kLimit = 2000000000ll;            // about a second at the boost clock
    extern __shared__ __align__(1024) unsigned char smem_dyn[];
    const uint32_t raw = smem_u32(smem_dyn);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* base_ptr = smem_dyn + (base - raw);
    const uint32_t bars = base + L::bar_off, abort_flag = bars + 16u * NST;
    auto full = [&](int s) { return bars + 8u * (uint32_t)s; };
    auto empty = [&](int s) { return bars + 8u * (uint32_t)(NST + s); };
    const int tid = threadIdx.x, lane = tid & 31;

    auto issue = [&](int t, int stage) {
        const int c0 = (t % col_tiles) * kQT, r0 = (t / col_tiles) * kQT;
        const uint32_t dst = base + L::in_off + (uint32_t)stage * L::in_stage;
        mbar_expect_tx(full(stage), L::in_stage);
        if constexpr (OCT) {
#pragma unroll 1
            for (int k = 0; k < 8; ++k)
                tma_load_2d(dst + (uint32_t)k * kOctClass, &tmX, full(stage), (int)(((int64_t)k * ldx + c0) & ~7ll), r0 / 8);
        } else {
            tma_load_2d(dst, &tmX, full(stage), c0, r0);
            tma_load_2d(dst + kQT * 128, &tmX, full(stage), c0 + 64, r0);
        }
    };
    if (tid == 0) {
        for (int s = 0; s < NST; ++s) {
            mbar_init(full(s), SHIFT ? NT : 1);
            mbar_init(empty(s), NT);
        }
        sts_u32(abort_flag, 0u);
        mbar_fence_init();
        fence_proxy_async_smem();
    }
    after_predecessor();
    ShiftLoader<NT> loader;
    if constexpr (SHIFT) {
        loader.x = static_cast<const unsigned char*>(x);
        loader.pitch = ldx * 2;
        loader.R = R;
        loader.C = C;
        if ((int)blockIdx.x < num_tiles) loader.request(tid, ((int)blockIdx.x / col_tiles) * kQT, ((int)blockIdx.x % col_tiles) * kQT);
    } else if (tid == 0) {
        for (int s = 0; s < NST - 1; ++s) {
            const int64_t t0 = (int64_t)blockIdx.x + (int64_t)s * gridDim.x;
            if (t0 < num_tiles) issue((int)t0, s);
        }
    }
    __syncthreads();
    if constexpr (SHIFT) {
        if ((int)blockIdx.x < num_tiles) {
            loader.store(tid, ((int)blockIdx.x / col_tiles) * kQT, ((int)blockIdx.x % col_tiles) * kQT, base + L::in_off);
            mbar_arrive(full(0));
        }
    }

    const bool col_role = tid < kQThreads;
    const int rt_id = col_role ? 1 : 2;                   // the role's named barrier
    const int rtid = col_role ? tid : tid - kQThreads;    // thread index inside the role
    int fail_code = 0;
    bool ok = true;
    int it = 0, cur = 0;
    uint32_t par = 0;                                      // parity of stage `cur`'s full barrier for this use
    for (int64_t t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it) {
        const int64_t tnext = t + gridDim.x;
        if constexpr (SHIFT) {
            if (tnext < num_tiles) loader.request(tid, (int)(tnext / col_tiles) * kQT, (int)(tnext % col_tiles) * kQT);
        } else if (tid == 0) {
            // the tile NST - 1 iterations ahead goes into the stage that was read in the previous iteration
            const int64_t tn = t + (int64_t)(NST - 1) * gridDim.x;
            if (tn < num_tiles) {
                const int sn = cur == 0 ? NST - 1 : cur - 1;
                if (it >= 1) ok = mbar_wait(empty(sn), (uint32_t)(((it - 1) / NST) & 1), abort_flag, kLimit);
                if (ok) issue((int)tn, sn);
                else fail_code = QW_EMPTY;
            }
        }
        if (ok) {
            ok = mbar_wait(full(cur), par, abort_flag, kLimit);
            if (!ok) fail_code = QW_LOAD;
        }
        const int c0 = (int)(t % col_tiles) * kQT, r0 = (int)(t / col_tiles) * kQT;
        const uint32_t in_tile = base + L::in_off + (uint32_t)cur * L::in_stage;
        // kOct: elements between the class's first fetched column and the tile's
        auto oct_shift = [&](int k) { return ((uint32_t)k * (uint32_t)ldx + (uint32_t)c0) & 7u; };
        const int this_stage = cur;
        if (++cur == NST) { cur = 0; par ^= 1u; }
        // SHIFT: the next tile goes into stage `cur`, last read NST - 1 iterations ago
        auto store_next = [&] {
            if constexpr (SHIFT) {
                if (tnext < num_tiles) {
                    if (ok && it >= NST - 1) {
                        ok = mbar_wait(empty(cur), (uint32_t)(((it + 1 - NST) / NST) & 1), abort_flag, kLimit);
                        if (!ok) fail_code = QW_EMPTY;
                    }
                    // warp-aligned: the lanes exchange bytes; after a wait that ran out nothing is stored
                    ok = __all_sync(0xffffffffu, ok);
                    if (ok) {
                        loader.store(tid, (int)(tnext / col_tiles) * kQT, (int)(tnext % col_tiles) * kQT, base + L::in_off + (uint32_t)cur * kInStage);
                        mbar_arrive(full(cur));
                    }
                }
            }
        };

        if (col_role) {
            // ---------------- column-wise ----------------
            const int p = rtid & 63, g = rtid >> 6;        // column pair, group of 32 rows
            const int h = p >> 5, w = p & 31;              // sub-tile and word of the 128-byte row
            const uint32_t in = in_tile + (uint32_t)(h * kQT * 128) + (uint32_t)((w & 3) * 4);
            uint32_t v[32];
            uint32_t m2 = 0u;
            if (ok) {
                if constexpr (OCT) {
                    const int valid = C - (c0 + 2 * p);    // columns of the pair inside the tensor
                    const uint32_t keep = valid >= 2 ? 0xffffffffu : valid == 1 ? 0xffffu : 0u;
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const uint32_t sh = oct_shift(k);
                        const uint32_t at = in_tile + (uint32_t)k * kOctClass + (uint32_t)(g * 4) * kOctRow + (sh >> 1) * 4u + (uint32_t)p * 4u;
#pragma unroll
                        for (int j = 0; j < 4; ++j) v[8 * j + k] = lds_u32(at + (uint32_t)j * kOctRow);
                        if (sh & 1u) {
#pragma unroll
                            for (int j = 0; j < 4; ++j) v[8 * j + k] = __funnelshift_r(v[8 * j + k], lds_u32(at + (uint32_t)j * kOctRow + 4u), 16);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        v[i] &= keep;
                        m2 = Pk<T>::absmax(v[i], m2);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const int r = g * 32 + i;
                        v[i] = lds_u32(in + swz(r, w >> 2));
                        m2 = Pk<T>::absmax(v[i], m2);
                    }
                }
                mbar_arrive(empty(this_stage));            // this thread's part of the stage is in registers
            }
            float alo, ahi;
            Pk<T>::unpack(m2, alo, ahi);
            float2* ex = reinterpret_cast<float2*>(base_ptr + L::ex_off);
            if (B > 32) ex[g * 64 + p] = make_float2(alo, ahi);
            // the previous tile's store must have read the output tile before it is written again
            if (rtid == 0) tma_store_wait_read();
            ok = role_barrier_all(rt_id, kQThreads, ok);
            if (!ok) break;
            if (B > 32) {
                constexpr int GPB = B / 32;                // row groups per block
                const int g0 = (g / GPB) * GPB;
#pragma unroll
                for (int k = 0; k < GPB; ++k) {
                    const float2 o = ex[(g0 + k) * 64 + p];
                    alo = fmaxf(alo, o.x);
                    ahi = fmaxf(ahi, o.y);
                }
            }
            PairQ pq;
            pq.set(alo, ahi);
            const int c = 2 * p;
            float sum_lo = 0.0f, sum_hi = 0.0f;            // SUM: this thread's 32 rows of both columns
            const uint32_t outc = base + L::outc_off;
            auto quantize_cols = [&](auto way_tag) {
                constexpr int WAY = decltype(way_tag)::value;
#pragma unroll
                for (int part = 0; part < 2; ++part) {     // 16 rows = one 16-byte piece of each column's output row
                    uint32_t wl[4], wh[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        uint32_t bl[4], bh[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            float xlo, xhi;
                            Pk<T>::unpack(v[part * 16 + k * 4 + u], xlo, xhi);
                            if (SUM) {
                                sum_lo += xlo;
                                sum_hi += xhi;
                            }
                            pq.template q<WAY>(xlo, xhi, bl[u], bh[u]);
                        }
                        wl[k] = pack4(bl[0], bl[1], bl[2], bl[3]);
                        wh[k] = pack4(bh[0], bh[1], bh[2], bh[3]);
                    }
                    sts_v4(outc + swz(c, g * 2 + part), wl[0], wl[1], wl[2], wl[3]);
                    sts_v4(outc + swz(c + 1, g * 2 + part), wh[0], wh[1], wh[2], wh[3]);
                }
            };
            pq.template choose<T, DUAL && IN == kTiled, FIVE>(quantize_cols);
            // scales [ceil(R/B), C]: the first row group of each block writes the pair
            if ((g % (B / 32)) == 0) {
                const int rb = r0 + g * 32;
                if (rb < R && c0 + c < C) {
                    float* dst = s_col + (int64_t)(rb / B) * C + c0 + c;
                    if (c0 + c + 1 < C && (reinterpret_cast<uintptr_t>(dst) & 7u) == 0) {
                        *reinterpret_cast<float2*>(dst) = make_float2(alo, ahi);
                    } else {
                        dst[0] = alo;
                        if (c0 + c + 1 < C) dst[1] = ahi;
                    }
                }
            }
            if (SUM) reinterpret_cast<float2*>(base_ptr + L::sum_off)[g * 64 + p] = make_float2(sum_lo, sum_hi);
            fence_proxy_async_smem();
            role_barrier(rt_id, kQThreads);
            if (rtid == 0) {
                tma_store_2d(&tmQc, outc, r0, c0);
                tma_store_commit();
            }
            if (SUM && rtid < kQT && c0 + rtid < C) {
                // the tile's row groups in ascending order; the next tile writes them behind another barrier of the role
                const float* part = reinterpret_cast<const float*>(base_ptr + L::sum_off) + rtid;
                sums[(int64_t)(r0 / kQT) * C + c0 + rtid] = ((part[0] + part[kQT]) + part[2 * kQT]) + part[3 * kQT];
            }
            store_next();
        } else {
            // ---------------- row-wise ----------------
            const int rwarp = rtid >> 5;
            // kOct: warp w has the rows equal to w modulo 8, in the order of their place in the staged class
            const int row = OCT ? (lane & 15) * 8 + rwarp : rwarp * 16 + (lane & 7) + 8 * (lane >> 4), half = OCT ? lane >> 4 : (lane >> 3) & 1;
            const int srow = OCT ? rwarp * 16 + (lane & 15) : row;        // row of the staged output
            const uint32_t in = in_tile + (uint32_t)(half * kQT * 128);
            uint32_t v[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0u;
            if (ok) {
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const uint32_t at = OCT ? in_tile + (uint32_t)rwarp * kOctClass + (uint32_t)(lane & 15) * kOctRow + (uint32_t)(half * 128 + 16 * k) : in + swz(row, k);
                    lds_v4(at, v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
                }
                if constexpr (OCT) {
                    uint32_t t[4];
                    lds_v4(in_tile + (uint32_t)rwarp * kOctClass + (uint32_t)(lane & 15) * kOctRow + (uint32_t)(half * 128 + 128), t[0], t[1], t[2], t[3]);
                    const uint32_t sh = oct_shift(rwarp), bits = (sh & 1u) * 16u;
                    auto shifted = [&](auto words) {       // the columns begin `WS` words and `bits` bits into what was read
                        constexpr int WS = decltype(words)::value;
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            v[i] = __funnelshift_r(i + WS < 32 ? v[(i + WS) & 31] : t[(i + WS) & 3], i + WS + 1 < 32 ? v[(i + WS + 1) & 31] : t[(i + WS + 1) & 3], bits);
                    };
                    if ((sh >> 1) == 0) shifted(std::integral_constant<int, 0>{});
                    else if ((sh >> 1) == 1) shifted(std::integral_constant<int, 1>{});
                    else if ((sh >> 1) == 2) shifted(std::integral_constant<int, 2>{});
                    else shifted(std::integral_constant<int, 3>{});
                    const int valid = C - (c0 + half * 64);
                    if (valid < 64) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = 2 * i >= valid ? 0u : 2 * i + 1 >= valid ? v[i] & 0xffffu : v[i];
                    }
                }
                mbar_arrive(empty(this_stage));
            }
            constexpr int NBT = B == 32 ? 2 : 1;           // blocks inside the thread's 64 columns
            float amax[NBT];
#pragma unroll
            for (int b = 0; b < NBT; ++b) {
                uint32_t m2 = 0u;
#pragma unroll
                for (int i = 0; i < 32 / NBT; ++i) m2 = Pk<T>::absmax(v[b * (32 / NBT) + i], m2);
                float lo, hi;
                Pk<T>::unpack(m2, lo, hi);
                amax[b] = fmaxf(lo, hi);
            }
            if (B == 128) amax[0] = fmaxf(amax[0], __shfl_xor_sync(0xffffffffu, amax[0], OCT ? 16 : 8));   // the row's other half
            if (rtid == 0) tma_store_wait_read();
            ok = role_barrier_all(rt_id, kQThreads, ok);
            if (!ok) break;
            const uint32_t outr = base + L::outr_off;
#pragma unroll
            for (int b = 0; b < NBT; ++b) {
                PairQ pq;
                pq.set(amax[b], amax[b]);
                auto quantize_row = [&](auto way_tag) {
                    constexpr int WAY = decltype(way_tag)::value;
#pragma unroll
                    for (int k = 0; k < 4 / NBT; ++k) {
                        uint32_t wd[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int i = b * (32 / NBT) + k * 8 + u * 2;
                            float x0, x1, x2, x3;
                            uint32_t b0, b1, b2, b3;
                            Pk<T>::unpack(v[i], x0, x1);
                            Pk<T>::unpack(v[i + 1], x2, x3);
                            pq.template q<WAY>(x0, x1, b0, b1);
                            pq.template q<WAY>(x2, x3, b2, b3);
                            wd[u] = pack4(b0, b1, b2, b3);
                        }
                        sts_v4(outr + swz(srow, half * 4 + b * (4 / NBT) + k), wd[0], wd[1], wd[2], wd[3]);
                    }
                };
                pq.template choose<T, DUAL && IN == kTiled, FIVE>(quantize_row);
            }
            // scales [ceil(C/B), R] (transposed): eight consecutive rows per quarter-warp
            if (r0 + row < R) {
#pragma unroll
                for (int b = 0; b < NBT; ++b) {
                    const int col = c0 + half * 64 + b * 32;
                    if (col < C && !(B == 128 && half == 1)) s_row[(int64_t)(col / B) * R + r0 + row] = amax[b];
                }
            }
            fence_proxy_async_smem();
            role_barrier(rt_id, kQThreads);
            if (rtid == 0) {
                if constexpr (OCT) tma_store_3d(&tmQr, outr, c0, r0 / 8, 0);
                else tma_store_2d(&tmQr, outr, c0, r0);
                tma_store_commit();
            }
            store_next();
        }
    }
    // shared memory must stay valid until the last stores have read it
    if (rtid == 0) tma_store_wait_read();
    if (!ok && rtid == 0 && fail_code != 0) report_timeout(status, abort_flag, fail_code);
}

// int8 [rows, cols] row-major, row pitch ld bytes (a multiple of 16, 16-byte aligned base) -> boxes of 128 x 128 bytes, 128-byte swizzle
int make_q_map(CUtensorMap* map, int8_t* ptr, int64_t rows, int64_t cols, int64_t ld) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(BI8_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    ensure_current_context();
    cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t gstride[1] = {(cuuint64_t)ld};
    cuuint32_t box[2] = {128, 128};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, ptr, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(BI8_ERR_CUDA, "cuTensorMapEncodeTiled (int8 tile) failed with CUresult %d", (int)r);
    return BI8_OK;
}

// The same tensor as [8 rows modulo 8][rows / 8][cols] -> boxes of 8 x 16 rows x 128 bytes (rows a multiple of 8)
int make_q_oct_map(CUtensorMap* map, int8_t* ptr, int64_t rows, int64_t cols, int64_t ld) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(BI8_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    ensure_current_context();
    cuuint64_t gdim[3] = {(cuuint64_t)cols, (cuuint64_t)(rows / 8), 8};
    cuuint64_t gstride[2] = {(cuuint64_t)ld * 8, (cuuint64_t)ld};
    cuuint32_t box[3] = {128, kQT / 8, 8};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, ptr, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(BI8_ERR_CUDA, "cuTensorMapEncodeTiled (int8 rows modulo 8) failed with CUresult %d", (int)r);
    return BI8_OK;
}

// 16-bit [rows, cols] with rows of any even alignment and row pitch ld elements, rows a multiple of 8 and a 16-byte aligned base, as
// "rows" of eight rows -> boxes of 136 columns x 16 of them, no swizzle.  Columns behind a row are the next row's.
int make_x_oct_map(CUtensorMap* map, const void* ptr, int64_t rows, int64_t cols, int64_t ld) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(BI8_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    ensure_current_context();
    cuuint64_t gdim[2] = {(cuuint64_t)(7 * ld + cols), (cuuint64_t)(rows / 8)};
    cuuint64_t gstride[1] = {(cuuint64_t)ld * 16};
    cuuint32_t box[2] = {kOctCols, kQT / 8};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(ptr), gdim, gstride, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(BI8_ERR_CUDA, "cuTensorMapEncodeTiled (input rows modulo 8) failed with CUresult %d", (int)r);
    return BI8_OK;
}

// 16-bit [rows, cols] row-major with row pitch ld elements -> boxes of 64 columns x 128 rows, 128-byte swizzle
int make_x_map(CUtensorMap* map, const void* ptr, int64_t rows, int64_t cols, int64_t ld) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(BI8_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    ensure_current_context();
    cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t gstride[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {64, 128};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(ptr), gdim, gstride, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(BI8_ERR_CUDA, "cuTensorMapEncodeTiled (input tile) failed with CUresult %d", (int)r);
    return BI8_OK;
}

// Encoded maps are looked up in the library's map table first (kinds 5 and 6 there): a training step quantizes tensors of
// the same few shapes at addresses the allocator keeps handing back, and an encode is a driver call of a few microseconds.
int cached_x_map(CUtensorMap* map, int dev, const void* ptr, int64_t rows, int64_t cols, int64_t ld, bool oct) {
    const MapKey key{dev, oct ? 7 : 5, ptr, rows, cols, ld, 128, 64};
    if (map_cache().find(key, map)) return BI8_OK;
    const int rc = oct ? make_x_oct_map(map, ptr, rows, cols, ld) : make_x_map(map, ptr, rows, cols, ld);
    if (rc == BI8_OK) map_cache().put(key, *map);
    return rc;
}
int cached_q_map(CUtensorMap* map, int dev, int8_t* ptr, int64_t rows, int64_t cols, int64_t ld, bool oct) {
    const MapKey key{dev, oct ? 8 : 6, ptr, rows, cols, ld, 128, 128};
    if (map_cache().find(key, map)) return BI8_OK;
    const int rc = oct ? make_q_oct_map(map, ptr, rows, cols, ld) : make_q_map(map, ptr, rows, cols, ld);
    if (rc == BI8_OK) map_cache().put(key, *map);
    return rc;
}

template <typename T, int B, bool DUAL, int IN, bool SUM, bool FIVE = false>
int launch_tile(const CUtensorMap& tx, const CUtensorMap& tqc, const CUtensorMap& tqr, const void* x, int64_t ldx, float* s_col, float* s_row, float* sums,
                int64_t R, int64_t C, cudaStream_t st) {
    const int64_t ctiles = (C + kQT - 1) / kQT, rtiles = (R + kQT - 1) / kQT;
    if (ctiles * rtiles >= (1ll << 31)) return fail(BI8_ERR_SHAPE, "quantize: grid too large");
    constexpr size_t smem = (DUAL ? QLayout<3, IN>::bytes_dual : QLayout<2, IN>::bytes_col) + 1024;
    static SmemOptIn opt_in;
    const int rc = opt_in.ensure(quantize_tile_kernel<T, B, DUAL, IN, SUM, FIVE>, smem);
    if (rc != BI8_OK) return rc;
    int* status = device_status_ptr();
    if (!status) return BI8_ERR_CUDA;
    const DeviceInfo di = device_info();
    const int64_t tiles = ctiles * rtiles;
    const int64_t resident = (int64_t)(DUAL ? 1 : 2) * di.sms;                 // CTAs that fit at once
    const int grid = (int)(tiles < resident ? tiles : resident);
    return launch_chained(quantize_tile_kernel<T, B, DUAL, IN, SUM, FIVE>, grid, DUAL ? 2 * kQThreads : kQThreads, smem, st, tx, tqc, tqr, x, ldx, s_col, s_row, sums, (int)R, (int)C, (int)ctiles, (int)tiles, status);
}

// The column-wise kernel's way with bf16.  One operation per pair is faster until the memory is what bounds it; there warps that ask for it in shorter
// bursts get less of it (both ways in a graph, one / five, block 64, blocks 32 and 128 alike).  Tiles by tensor map: 8192 x 8192 35.5 / 36.3 us, 8192 x
// 10240 43.7 / 43.4, 8192 x 12288 51.8 / 51.7, 8192 x 14336 61.9 / 59.8, 16384 x 16384 154.5 / 144.4.  By every eighth row: 8192 x 30001 129 / 136, 8192 x
// 35001 148-153 / 157, 32768 x 10001 167 / 180, 16384 x 20001 170-190 / 179, 8192 x 40001 184 / 177, 65536 x 6001 238 / 215, 8192 x 50257 240 / 221.
constexpr int64_t kFiveTiled = 160ll << 20, kFiveOct = 624ll << 20;         // bytes of the input
template <typename T>
bool five_operations(int64_t R, int64_t C, bool tiled) {
    return std::is_same_v<T, __nv_bfloat16> && R * C * 2 >= (tiled ? kFiveTiled : kFiveOct);
}

template <typename T>
int tile_dispatch(const void* x, int64_t ldx, int8_t* q_col, int64_t ldqc, float* s_col, int8_t* q_row, int64_t ldqr, float* s_row, float* sums, int64_t R,
                  int64_t C, int block, cudaStream_t st) {
    CUtensorMap tx, tqc, tqr;
    int dev = 0;
    BI8_CUDA_TRY(current_device(&dev));
    int rc = cached_q_map(&tqc, dev, q_col, C, R, ldqc, false);
    if (rc != BI8_OK) return rc;
    tx = tqr = tqc;
    const bool tiled = aligned(x, 16) && (ldx * 2) % 16 == 0;         // a tensor map can describe the input
    const bool oct = !tiled && aligned(x, 16) && R % 8 == 0 && ldx < (1ll << 28);   // ... or every eighth row of it
    if (tiled || oct) {
        rc = cached_x_map(&tx, dev, x, R, C, ldx, oct);
        if (rc != BI8_OK) return rc;
    }
    const bool dual = q_row != nullptr;
    if (dual) {
        rc = cached_q_map(&tqr, dev, q_row, R, C, ldqr, oct);
        if (rc != BI8_OK) return rc;
    }
    constexpr bool BF = std::is_same_v<T, __nv_bfloat16>;
    const bool five = five_operations<T>(R, C, tiled);
#define BI8_TILE_C(BB)                                                                                           \
    five && tiled ? launch_tile<T, BB, false, kTiled, false, BF>(tx, tqc, tqr, x, ldx, s_col, s_row, sums, R, C, st) \
    : five && oct ? launch_tile<T, BB, false, kOct, false, BF>(tx, tqc, tqr, x, ldx, s_col, s_row, sums, R, C, st)   \
                  : BI8_TILE_D(BB, false, false)
#define BI8_TILE_D(BB, DUAL, SUM)                                                                                \
    tiled ? launch_tile<T, BB, DUAL, kTiled, SUM>(tx, tqc, tqr, x, ldx, s_col, s_row, sums, R, C, st)           \
    : oct ? launch_tile<T, BB, DUAL, kOct, SUM>(tx, tqc, tqr, x, ldx, s_col, s_row, sums, R, C, st)             \
          : launch_tile<T, BB, DUAL, kShift, SUM>(tx, tqc, tqr, x, ldx, s_col, s_row, sums, R, C, st)
#define BI8_TILE(BB) \
    if (block == BB) return !dual ? (BI8_TILE_C(BB)) : sums ? (BI8_TILE_D(BB, true, true)) : (BI8_TILE_D(BB, true, false));
    BI8_TILE(32) BI8_TILE(64) BI8_TILE(128)
#undef BI8_TILE
#undef BI8_TILE_C
#undef BI8_TILE_D
    return fail(BI8_ERR_BLOCK, "tile quantizer supports block 32, 64, 128 (got %d)", block);
}

}  // namespace

// The tile quantizer takes 16-bit inputs of any alignment; its int8 outputs leave by TMA and need 16-byte aligned bases and row
// pitches (ldqc for the transposed one, ldqr for the row-wise one).
bool quantize_tile_applicable(int dt, const void* q_col, int64_t ldqc, const void* q_row, int64_t ldqr, int64_t R, int64_t C, int block) {
    if (dt != BI8_BF16 && dt != BI8_F16) return false;
    if (block != 32 && block != 64 && block != 128) return false;
    if (R <= 0 || C <= 0 || R >= (1ll << 31) - 256 || C >= (1ll << 31) - 256) return false;
    if (!aligned(q_col, 16) || ldqc % 16 != 0) return false;
    if (q_row != nullptr && (!aligned(q_row, 16) || ldqr % 16 != 0)) return false;
    return device_info().ok;
}

int launch_quantize_tile(const void* x, int dt, int64_t ldx, int8_t* q_col, int64_t ldqc, float* s_col, int8_t* q_row, int64_t ldqr,
                         float* s_row, int64_t R, int64_t C, int block, cudaStream_t st, float* sums) {
    if (dt == BI8_BF16) return tile_dispatch<__nv_bfloat16>(x, ldx, q_col, ldqc, s_col, q_row, ldqr, s_row, sums, R, C, block, st);
    if (dt == BI8_F16) return tile_dispatch<__half>(x, ldx, q_col, ldqc, s_col, q_row, ldqr, s_row, sums, R, C, block, st);
    return fail(BI8_ERR_DTYPE, "tile quantizer takes bf16 or fp16 input");
}

}  // namespace bi8
