// Int8 block GEMM with fused dequantize on the sm_100a tensor cores.
//
// Replaces the reference kernel at triton_functions.py:69-139 (path inside the reference project):
//   P_j = A[:, jB:(j+1)B] . Bt[:, jB:(j+1)B]^T      exact int32 (line 115)
//   acc += sB[j,n] * sA[j,m] * float(P_j) / 127^2   fp32, j ascending (line 120)
//   C = cast(acc) (+ cast(bias))                    (lines 125-131)
//
// One persistent CTA per SM works on 128 x BN output tiles.  Warp roles:
//   warp 0      producer.  Per stage two TMA copies of 128-byte-swizzled K-major operand tiles (A: 128 rows, Bt: BN
//               rows, 128 K-bytes) into a ring of kStages slots, and two TMA copies of the stage's block scales (fp32
//               boxes [blocks, 128] of sA and [blocks, BN] of sB), all four on the stage's one "full" barrier.  Scale tensors that a
//               tensor map cannot describe (base or row length not 16-byte aligned) are
//               copied with cp.async by the warp's 32 lanes instead, arriving on the same barrier.  sA lies in the operand stage's slot:
//               only the seeder reads it, and the slot is free when the stage's MMAs are complete and the seeder has
//               arrived (EMPTY_AB).  sB lies in a ring of its own without barriers: the promotion warps read a stage's column scales after they
//               have seen one of its accumulators complete (the MMAs were issued after the stage's barrier), and the ring is deep
//               enough that a slot is never rewritten while in use (SC_STAGES).
//   warp 1      issues tcgen05.mma kind::i8 (M128 N=BN K32): the MMAs of one quantisation block accumulate into one of
//               three s32 accumulators in tensor memory, then a commit hands that accumulator to the promotion warps.
//   warp 2      seeder: puts the seed pattern (below) into every accumulator that the promotion warps have released, and makes the row
//               records of every stage: per row and block (s, -1.5*2^23*s), s the row scale as the fold takes it.
//   warp 3      storer: moves finished tiles from shared memory to C by TMA stores.
//   warps 4-19  promotion, four warps per tensor-memory lane quarter.  A warp owns 32 rows x 40 columns of the tile.  Per
//               block it reads its part of the finished accumulator, folds the values into fp32 accumulators in registers, and
//               releases the accumulator as soon as the last columns are in registers.  After the last block of a tile it casts, adds
//               the bias, stages its 32 x 40 part in shared memory, adds the residual there and goes on with the next tile.
// What bounds the kernel: the promotion, t = P*s_row and acc += s_col*t for two columns per FFMA2, and what its warps issue beside it.  A
// scheduler takes two cycles per FFMA2 and one per other instruction, and each of its four warps has 40 and about 50 of them per block (92
// instructions a block and promotion warp in all, epilogue and role warps included): 520 cycles
// (the promotion alone, without MMAs; 372 without the barriers).  MMAs beside it cost another 60 to 70 cycles each: one of M128 N160 K32 reads
// 9.2 KB of operands in 80 cycles, 90 % of the shared memory's bandwidth, and the loads of the scales wait (552, 602 and 733 cycles a block
// of 32, 64 and 128; without the loads of scales 604 at 128).  The MMAs and seeds alone take 162, 242 and 402.  Every register that a
// shared-memory load fills takes its time on that pipe, broadcast or not.  As a thread with one row and 40
// columns (32x32b reads) a warp loaded 41 scales per block and thread; with four rows and ten columns (16x256b) 4 records and 10 scales,
// each scale pair of the columns used for four rows in turn.  Row scales are prepared once per CTA by the seeder, not by every
// thread for its four rows.  At 128 the operands' way from L2 (64 bytes per cycle and SM, 576 cycles per 128 x 160 x 128) bounds as well.
// 8192 x 4096 x 11008, cold: 672 -> 591 us at block 64, 425 -> 383 at 128, 1327 -> 1177 at 32 (with the row-wise reads and the
// issuer as a loop of its warp, the same GPU; others take 1 to 2 % more on either side); a lab loop without epilogue 683 -> 535, 731 -> 569 and 611 -> 535 cycles a block.
// Reading 8 + 32 columns at a time, the accumulator is free early and the first fold hides the second read: in that loop 527 cycles
// against 548 for all at once, 536 for 16 + 24, 636 for five times eight.
// The release of an accumulator is one predicated arrival (a branch around it: 577 cycles a block, 538 so), and the issuer tests a stage and its first
// accumulator at once: sustained 681 -> 672 us at block 64, 1182 -> 1160 at 32, 240 = 240 for 2048 x 4096 x 22016 at 128.
// One read for 32 columns of a half instead of two: 672.8 -> 670.5 us, 1175 -> 1168; 8192 x 768 x 50257 779.5 -> 772.5.
// Slower: a loop of whole cycles of three blocks with the rest behind it (8192 x 768 x 50257 777 -> 804, though fp32 4096^3 146 -> 141); the next block's words, or words and scales, requested behind this block's folds (649 us cold at block 64 against 614); records of 16 bytes
// that need no moves (655 cycles against 561) or of 4 bytes (591); two wide warps per quarter with everything requested a block ahead (660 cycles
// against 602); row records by the storer or the producer (613 to 900 us against 601).
//
// Registers: a scheduler (SM sub-partition) owns a quarter of the register file and every fourth warp, and setmaxnreg can
// only move registers between warps of the same scheduler.  Each scheduler has exactly one of warps 0-3, which shrinks,
// and four promotion warps, which grow: 96 at launch -> 32 and 112.
//
// Seeded conversion (default): every accumulator starts as the bit pattern of 1.5*2^23 and the MMAs accumulate on top
// of it.  Integer addition on that pattern is exact float arithmetic while |P| < 2^22 (127^2 * 128 < 2^22), so the word
// read back is the float 1.5*2^23 + P and
//   t = fma(word, s, -1.5*2^23 * s) = fl(P * s)
// needs no int->float conversion.  s = sA[j,m]/127^2 rounded to 22 significant bits makes 1.5*2^23*s exact.
// The pattern is written by an fp16 MMA of constants (every row 2048, 2048, 2048, 0 ...: 3 * 2048^2 = 1.5*2^23, exact in any
// order) that overwrites the accumulator, issued by the seeder and complete (commit, barrier) before the block's int8 MMAs are
// issued; its A lies in tensor memory, so that it reads only B from shared memory (1.3 % at block 64: 678 -> 668 us).  As
// tensor-memory stores of the promotion warps it cost them 100 of 590 cycles per block in isolation and held every accumulator
// until the last of its columns was folded.
#include "bi8_common.cuh"
#include "tc_common.cuh"

#include <cstdint>
#include <cstring>
#include <mutex>
#include <type_traits>

namespace bi8 {
namespace {

using namespace ptx;

constexpr int kBM = 128;                 // tile rows
constexpr int kAccBufs = 3;              // s32 accumulators in tensor memory
constexpr int kProbeN = 256;             // N of the issue-rate probe's MMAs
constexpr int kStages = 4;               // operand stages of 128 K-bytes in flight
constexpr int kRoleWarps = 4;            // producer, MMA issuer, seeder, storer: one warp per scheduler gives its registers away
constexpr uint32_t kABytes = kBM * kBK;  // 16 KiB
constexpr uint32_t kSeedBits = 0x4B400000u;   // float 1.5 * 2^23
constexpr float kSeedF = 12582912.0f;

// Promotion warps per tensor-memory lane quarter, and what follows from it: a warp owns COLS columns of its 32 rows, a thread COLS results
// (a quarter of those columns in four rows).  (Two or three
// warps with 80 or 48 columns each were 7-18 % slower.)
constexpr int kPW = 4;
struct Cfg {
    static constexpr int BN = 160;                        // tile columns: kAccBufs * BN <= 512 tensor-memory columns
    static constexpr int COLS = BN / kPW;                 // columns owned by one promotion warp
    static constexpr int EPI_WARPS = 4 * kPW;
    static constexpr int THREADS = (kRoleWarps + EPI_WARPS) * 32;
    static constexpr int LAUNCH_REGS = 96;                // 65536 / THREADS, rounded down to a multiple of 8
    static constexpr int ROLE_REGS = 32;
    static constexpr int EPI_REGS = 112;
    static constexpr uint32_t B_BYTES = BN * kBK;
    static constexpr uint32_t STAGE_BYTES = kABytes + B_BYTES;
    static constexpr uint32_t scale_off = kStages * STAGE_BYTES;
    // setmaxnreg moves registers inside a scheduler's share of the CTA's launch-time allocation: the total after the
    // moves must not exceed it, or setmaxnreg.inc blocks forever.  (The launcher also checks the register count the
    // compiler really chose for the kernel.)
    static_assert(ROLE_REGS + kPW * EPI_REGS <= (1 + kPW) * LAUNCH_REGS, "register budget of a scheduler exceeds its launch allocation");
    static_assert((1 + kPW) * 32 * LAUNCH_REGS <= 16384, "launch allocation exceeds a scheduler's register file");
    static_assert(kAccBufs * BN <= 512 && COLS % 8 == 0 && BN % 32 == 0, "tile geometry");
    __host__ __device__ static constexpr uint32_t a_off(int s) { return (uint32_t)s * STAGE_BYTES; }
    __host__ __device__ static constexpr uint32_t b_off(int s) { return a_off(s) + kABytes; }
};

// Transposes a 4 x 4 matrix whose rows are the arrays of four neighbouring lanes (c the lane's place among them).
__device__ __forceinline__ void transpose4(uint32_t (&v)[4], uint32_t c) {
#pragma unroll
    for (int d = 1; d <= 2; d <<= 1)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i & d) continue;
            const bool up = (c & (uint32_t)d) != 0u;
            const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + d], d);
            if (up) v[i] = got;
            else v[i + d] = got;
        }
}

// How a finished tile leaves: kTma, through the tensor map tmC (16-bit outputs by the storer warp, fp32 ones in two passes by the promotion
// warps: handing the halves over was 2 us slower where there is one round of tiles); kRows, by the storer warp to 16-bit
// outputs whose rows no tensor map can describe, but every eighth of which one can (store_rows); kOwn, by the promotion warps,
// to all others.
enum StoreMode { kTma = 0, kRows = 1, kOwn = 2 };
// Instances of the kernel by the way its tiles leave: code for the other ways, even where it is not executed, costs the K loop
// registers.  kAnyOut in the instance's place at block 32 / 64 / 128: kTma16 8192 x 4096 x 11008 +1.4 / 0.9 / 0.8 %, 4096 x 512 x 4096 +4.9 / 7.9 /
// 0 %; kTma16Add 2048 x 768 x 3072 +1.1 / 2.6 / 0 %; kOwn16 8192 x 4096 x 11005 with bias 0 / 0.6 / 0 %; kWide 8192 x 4096 x 11008 0 / 1.7 /
// 0.4 %, 4096 x 512 x 4096 +1.7 / 1.3 / 3 %.
enum OutKind { kAnyOut = 0, kSplit, kCluster, kTma16, kTma16Add, kRows16, kOwn16, kWide };

struct TcParams {
    const float* sA;
    const float* sB;
    const void* bias;
    void* C;
    int32_t* partials;
    int* status;
    int64_t ldc;
    int M, N, K, nb;
    int tiles_m, tiles_n;
    int out_dtype, bias_dtype;
    int vec_store;      // C base and row pitch allow 16-byte stores
    int store;          // how undivided tiles leave (StoreMode)
    FastDiv by_tiles_m;
    int tma_scales;     // bit 0: sA is described by the tensor map tmSA, bit 1: sB by tmSB
    int ksplit;         // > 1: the K stages are divided over ksplit work items per tile (split-K)
    int stages_per_split;
    float* ws;          // split-K: fp32 partial results, one slot of slot_floats values per work item (ws_index)
    int slot_floats;    // BN x the tile rows that exist in any tile, rounded up to the 32 of a warp
    const void* residual;     // [M, N] addend of the output type with row pitch ldr, or null
    int64_t ldr;
    int res_vec;        // its base and row pitch allow 16-byte loads
    unsigned wait_limit_us;   // 0: default limit of the bounded waits (about two seconds)
    int skip_stage;     // >= 0: diagnostic, the producer leaves this stage of its first work item out
};

template <int QB>
struct Geo {
    using C = Cfg;
    static constexpr int BPS = kBK / QB;                        // quantisation blocks per stage
    static constexpr int MMAS = QB / 32;                        // MMAs (K = 32) per block
    // Column scales: a ring of records of BN floats, one per block.  The producer fills the slot of stage s after the MMA warp has
    // committed stage s - kStages.  By then every promotion warp had released a block at most kAccBufs before that stage's last one (a tile
    // restarts on accumulator 0, so the use before may be up to five blocks back, but then a later block's release has been
    // seen), having read everything but some of the released block's scales: the oldest stage that may still be read is
    // s - kStages + 1 - ceil((kAccBufs + 1) / BPS) = s - SC_STAGES + 1, and the slot held s - SC_STAGES.
    static constexpr int SC_STAGES = kStages + (kAccBufs + 1 + BPS - 1) / BPS;
    static constexpr uint32_t SC_REC = C::BN * 4;               // bytes of a record
    static constexpr uint32_t SC_RING = SC_STAGES * BPS * SC_REC;
    static constexpr uint32_t sb_off = C::scale_off;
    // Row scales as they come, with the operand stage, and as the promotion warps read them: one (s, -1.5*2^23*s) per row and block,
    // made by the seeder warp.  That warp has seen the accumulator of the block before a stage released, and with it the records up to
    // kAccBufs blocks before that one read, when it writes a stage's.
    static constexpr uint32_t SA_STAGE = BPS * kBM * 4;
    static constexpr uint32_t sa_off = sb_off + SC_RING;
    static constexpr uint32_t ROW_REC = kBM * 8;
    static constexpr uint32_t ROW_RING = (BPS + kAccBufs) * ROW_REC;
    static constexpr uint32_t row_off = sa_off + kStages * SA_STAGE;
    static constexpr uint32_t bar_off = row_off + ROW_RING;
    // barrier slots (8 bytes each)
    static constexpr int FULL_AB = 0, EMPTY_AB = kStages, ACC_FULL = 2 * kStages, ACC_EMPTY = 2 * kStages + kAccBufs,
                         ACC_SEEDED = 2 * kStages + 2 * kAccBufs, OUT_FULL = 2 * kStages + 3 * kAccBufs, OUT_EMPTY = OUT_FULL + 1,
                         RX_FULL = OUT_EMPTY + 1, NBARS = RX_FULL + 8;
    static constexpr uint32_t misc_off = bar_off + NBARS * 8;   // tmem holder (4 B) + abort flag (4 B) + never-raised flag (4 B)
    // Finished tiles are staged as one part of 32 rows of 80 bytes per promotion warp; a tile of fp32 takes two passes of half its columns.
    static constexpr uint32_t PART_ROW = C::COLS * 2, PART_BYTES = 32 * PART_ROW;
    // kRows: [8 rows modulo 8][16] bodies of 304 bytes, then per row the first and the last eight elements
    static constexpr uint32_t BODY = C::BN * 2 - 16, CLASS_BYTES = kBM / 8 * BODY, EDGES = 8 * CLASS_BYTES;
    static constexpr uint32_t OUT_BYTES = EDGES + kBM * 32;
    // operand B of the seeding MMAs: 16 fp16 values per row, the same eight rows (two core matrices) for all of them
    static constexpr uint32_t seed_off = (misc_off + 16 + 127) & ~127u;
    static constexpr uint32_t SEED_BYTES = 256;
    // kCluster: what a warp has of a tile, in fp32; a warp that finishes its part receives one from every other CTA, and stages there
    static constexpr uint32_t RX_BYTES = 32 * C::COLS * 4;
    static constexpr uint32_t out_off = seed_off + SEED_BYTES;
    static constexpr uint32_t total = out_off + OUT_BYTES;
    static constexpr size_t cluster_total(int n) {
        const uint32_t rx = (uint32_t)((C::EPI_WARPS + n - 1) / n) * (uint32_t)(n - 1) * RX_BYTES;
        return out_off + (rx > OUT_BYTES ? rx : OUT_BYTES);
    }
    static_assert(PART_BYTES % 128 == 0 && CLASS_BYTES % 128 == 0 && OUT_BYTES >= C::EPI_WARPS * PART_BYTES && OUT_BYTES % 128 == 0, "TMA store sources are 128-byte aligned");
    static_assert(SC_REC % 128 == 0 && SA_STAGE % 128 == 0 && C::scale_off % 1024 == 0, "TMA destinations of the scale boxes are 128-byte aligned");
};

// Work item -> tile and K-stage range.  Items of one split are consecutive, so CTAs that run together work on different
// tiles of the same K range; the parts of a tile that a cluster shares are its CTAs.  `slot` is the item's place in the
// workspace, -1 where there is none.
template <int OUT>
__device__ __forceinline__ void item_range(int item, const TcParams& p, int nks, int& tile, int& slot, int& ks0, int& ks1) {
    if (OUT == kCluster) {
        tile = item / p.ksplit;
        const int split = item - tile * p.ksplit;
        slot = -1;
        ks0 = split * nks / p.ksplit;
        ks1 = (split + 1) * nks / p.ksplit;
    } else if (p.ksplit == 1) {
        tile = item;
        slot = -1;
        ks0 = 0;
        ks1 = nks;
    } else {
        const int tiles = p.tiles_m * p.tiles_n, split = item / tiles;
        tile = item - split * tiles;
        slot = tile * p.ksplit + split;
        ks0 = split * p.stages_per_split;
        ks1 = ks0 + p.stages_per_split < nks ? ks0 + p.stages_per_split : nks;
    }
}

template <int BN>
__device__ __forceinline__ void tile_coords(int tile, const TcParams& p, int& m0, int& n0) {
    // consecutive tiles (CTAs that run together) share a column panel of Bt and sweep the rows of A
    const int tn = (int)p.by_tiles_m.div((unsigned)tile);
    m0 = (tile - tn * p.tiles_m) * kBM;
    n0 = tn * BN;
}

// Bounded wait of a converged warp: one poll by every lane, then (phase not complete yet, or the lanes disagree) the
// bounded loop.  The result is the same in all lanes, so a warp-aligned instruction after the wait is never reached by
// only some of them.  (Not a function call: the callers run under different setmaxnreg budgets.)
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, uint32_t abort_flag, long long limit) {
    if (__builtin_expect(__all_sync(0xffffffffu, mbar_test(bar, parity)), 1)) return true;
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, limit));
}

// Blocks go round the kAccBufs = 3 accumulators and every stage has BPS blocks, so block `blk` of the stage at position
// `rot` in a cycle of three stages is block rot*BPS + blk of that cycle and uses accumulator (rot*BPS + blk) % 3.  A
// cycle of three stages ends where it began, on accumulator 0.
template <int BPS>
struct RotInfo {
    __host__ __device__ static constexpr int buf(int rot, int blk) { return (rot * BPS + blk) % kAccBufs; }
};

// A value the compiler must treat as unknown from here on.  Loop-invariant addresses of the promotion loop go through
// this: left alone, the compiler recomputes them (from the warp index, the thread index, the shared-memory base ...)
// inside every block instead of keeping a register, which costs more instructions than the fold itself has to spare.
__device__ __forceinline__ uint32_t keep(uint32_t v) {
    asm volatile("" : "+r"(v));
    return v;
}

// Folds the s32 words that a thread has read of NC columns from C0 on (one quantisation block; NC / 8 groups of four words for each half of
// 16 rows) into its fp32 accumulators: acc += sB[n] * (P * s), both products as packed FMAs on column pairs.  `sw` is the shared address
// of the block's first pair of column scales of this thread, s2 and n2 the scales of its four rows and their seed terms.
template <bool SEED, int NC, int C0, int COLS>
__device__ __forceinline__ void fold_columns(const uint32_t (&W)[NC], uint32_t sw, const uint64_t (&s2)[4], const uint64_t (&n2)[4], uint64_t (&acc2)[COLS / 2]) {
#pragma unroll
    for (int q = 0; q < NC / 8; ++q) {
        const uint64_t w = lds_b64(sw + (uint32_t)((C0 / 8 + q) * 32));
        uint64_t t[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint32_t* const S = W + (r >> 1) * (NC / 2) + 4 * q + 2 * (r & 1);
            if (SEED) {
                t[r] = fma_f32x2(pack_u32x2(S[0], S[1]), s2[r], n2[r]);
            } else {
                float sr, dup;
                unpack_f32x2(s2[r], sr, dup);
                t[r] = pack_f32x2(__fmul_rn((float)(int32_t)S[0], sr), __fmul_rn((float)(int32_t)S[1], sr));
            }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) acc2[C0 / 2 + 4 * q + r] = fma_f32x2(w, t[r], acc2[C0 / 2 + 4 * q + r]);
    }
}

// One whole 32-byte sector of a split-K part to and from L2.  As two 16-byte accesses each of a warp's 32 sectors crosses the
// L1-L2 path twice: 1.6 us per call on the storing side, 3-5 us on the loading side.
__device__ __forceinline__ void stg_v8(float* dst, const float (&f)[8]) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "f"(f[0]), "f"(f[1]), "f"(f[2]), "f"(f[3]), "f"(f[4]), "f"(f[5]),
                 "f"(f[6]), "f"(f[7])
                 : "memory");
}
__device__ __forceinline__ void ldcg_v8(float (&f)[8], const float* src) {
    asm volatile("ld.global.cg.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]), "=f"(f[4]), "=f"(f[5]), "=f"(f[6]), "=f"(f[7])
                 : "l"(src)
                 : "memory");
}

// Place of (lane quarter, column slice, group of eight columns, lane) in a workspace slot: a warp stores 1 KiB runs, a thread as one
// sector its two columns of four rows.
template <int COLS>
__host__ __device__ constexpr int ws_index(int quarter, int slice, int group, int lane) {
    return (((quarter * kPW + slice) * (COLS / 8) + group) * 32 + lane) * 8;
}

// element n of a vector of type `dt`
__device__ __forceinline__ float load_as_f32(const void* v, int dt, int64_t n) {
    if (dt == BI8_BF16) return __bfloat162float(static_cast<const __nv_bfloat16*>(v)[n]);
    if (dt == BI8_F16) return __half2float(static_cast<const __half*>(v)[n]);
    return static_cast<const float*>(v)[n];
}
// a + b where both have (a) or are first rounded to (b) the 16-bit type: the sum rounded once more (reference lines 127-131)
__device__ __forceinline__ uint32_t add_rounded(uint32_t a16, float b, bool bf) {
    if (bf) return pack_bf16x2(__fadd_rn(bf16lo(a16), __bfloat162float(__float2bfloat16_rn(b))), 0.0f) & 0xffffu;
    const float a = __half2float(__ushort_as_half((unsigned short)a16));
    return (uint32_t)__half_as_ushort(__float2half_rn(__fadd_rn(a, __half2float(__float2half_rn(b)))));
}

// One staged 16-byte piece (8 values of a 16-bit type or 4 of fp32) plus a vector of addends, value by value.
template <typename Addend>
__device__ __forceinline__ void add_piece(uint32_t addr, bool wide, bool bf, Addend addend) {
    uint32_t w[4];
    lds_v4(addr, w[0], w[1], w[2], w[3]);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        if (wide) w[u] = __float_as_uint(__fadd_rn(__uint_as_float(w[u]), addend(u)));
        else w[u] = add_rounded(w[u] & 0xffffu, addend(2 * u), bf) | (add_rounded(w[u] >> 16, addend(2 * u + 1), bf) << 16);
    }
    sts_v4(addr, w[0], w[1], w[2], w[3]);
}

// 32 staged rows of 16-bit elements to rows of odd length: a row's first 32 columns by the 32 lanes, then the columns behind them,
// several rows at once; running addresses, because a division and a product per element were more instructions than the
// promotion has (8192 x 50257, K 768: 1040 -> 902 us).  Not inlined: the registers of the K loop are to stay as they are.
template <int ROWB>
__device__ __forceinline__ void store_elements(unsigned char* dst, int64_t pitch, uint32_t stage, int lane, int rows, int cols) {
    constexpr int REST = ROWB / 2 - 32, ROWS = 32 / REST;
    static_assert(REST > 0 && 32 % REST == 0, "whole rows of remaining columns per step");
    auto column = [&](int r, int c, int step, int count) {
        if (c >= cols) return;
        unsigned char* d = dst + (int64_t)r * pitch + c * 2;
        uint32_t src = stage + (uint32_t)(r * ROWB + c * 2);
#pragma unroll 4
        for (int i = 0; i < count; ++i) {
            if (r + i * step < rows) *reinterpret_cast<uint16_t*>(d) = lds_u16(src);
            d += (int64_t)step * pitch;
            src += (uint32_t)step * ROWB;
        }
    };
    column(0, lane, 1, 32);
    column(lane / REST, 32 + lane % REST, ROWS, 32 / ROWS);
}

// A promotion warp's 32 staged rows of ROWB bytes to an output of any alignment: consecutive lanes store consecutive 4-byte words of a
// row, or 2-byte elements where the rows of a 16-bit output are not all 4-byte aligned.
template <int ROWB>
__device__ __noinline__ void store_own(unsigned char* dst, int64_t pitch, uint32_t stage, int rows_valid, int cols_left, bool wide, int lane) {
    const int cols_pass = ROWB / (wide ? 4 : 2);
    const int cols_valid = cols_left < cols_pass ? cols_left : cols_pass;      // rows_valid may exceed 32, both may be negative
    if (wide || (((reinterpret_cast<uintptr_t>(dst) | (uintptr_t)pitch) & 3u) == 0)) {
        constexpr int WPR = ROWB / 4;                          // words per staged row
        const int words = wide ? cols_valid : (cols_valid >> 1);
        const bool odd_tail = !wide && (cols_valid & 1) && cols_valid > 0;
#pragma unroll 4
        for (int idx = lane; idx < 32 * WPR; idx += 32) {
            const int r = idx / WPR, w = idx - r * WPR;
            if (r < rows_valid) {
                const uint32_t v = lds_u32(stage + (uint32_t)(idx * 4));
                unsigned char* d = dst + (int64_t)r * pitch + w * 4;
                if (w < words) *reinterpret_cast<uint32_t*>(d) = v;
                else if (odd_tail && w == words) *reinterpret_cast<uint16_t*>(d) = (uint16_t)(v & 0xffffu);
            }
        }
    } else {
        store_elements<ROWB>(dst, pitch, stage, lane, rows_valid, cols_valid);
    }
}

// 16-bit outputs with rows of any even alignment (kRows).  Rows that are eight apart have the same alignment, so a tensor map whose
// "rows" are eight rows long describes them: with h the elements of a tile row before its first 16-byte boundary, elements h .. h+151
// of the 16 rows of a tile that are equal modulo 8 leave by one TMA store, the first h and last 8-h one by one; a last, partial column of tiles is kOwn's.  8192 x 50257, K 768:
// 800 us by the promotion warps at block 64, 682 this way (545 with aligned rows); one bulk copy per row took 110 cycles a row, 16-byte pieces moved by
// the storer 190 (twice and nearly three times as long).  A thread's values are exchanged by shuffles first, so that a lane stages one row; words joined with the
// neighbouring lane's instead take 834 us, two-byte stores 953, an exchange through shared memory by stmatrix 703.
__device__ __forceinline__ uint32_t rows_head(const TcParams& p, uint32_t row_class, int n0) {
    return (0u - (row_class * (uint32_t)p.ldc + (uint32_t)n0)) & 7u;
}
// A thread's 40 results (pairs, in `e`) of slice `sl` of a row whose class has head `h` to the row's body and edges.
template <uint32_t BODY, int PAIRS>
__device__ __forceinline__ void stage_row(uint32_t body, uint32_t edges, uint32_t sl, uint32_t h, const uint32_t (&e)[PAIRS]) {
    if (sl == 0) sts_v4(edges, e[0], e[1], e[2], e[3]);
    if (sl == 3) sts_v4(edges + 16u, e[PAIRS - 4], e[PAIRS - 3], e[PAIRS - 2], e[PAIRS - 1]);
    // words of the body: at odd heads they hold the second half of one pair and the first of the next
    const uint32_t sh = (h & 1u) * 16u;
    const int at = (int)(sl * 4u * PAIRS) - 2 * (int)((h + 1u) & ~1u);        // byte of word 0 in the body
    const uint32_t dst = body + (uint32_t)at;
    if (sl != 0) {
        if (sh) sts_h(dst + 2u, e[0]);
        else sts_w(dst, e[0]);
        if (sh && sl != 3) sts_h(dst + 4u * PAIRS, e[PAIRS - 1] >> 16);
    } else {
        if (sh) sts_h(dst + 4u * PAIRS, e[PAIRS - 1] >> 16);
        if (at == 0) sts_w(dst, e[0]);
    }
#pragma unroll
    for (int k = 1; k < PAIRS; ++k) {
        const uint32_t v = __funnelshift_l(e[k - 1], e[k], sh);
        if (k < 4) {
            if (at + 4 * k >= 0) sts_w(dst + (uint32_t)(4 * k), v);
        } else if (k >= PAIRS - 4) {
            if (at + 4 * k < (int)BODY) sts_w(dst + (uint32_t)(4 * k), v);
        } else {
            sts_w(dst + (uint32_t)(4 * k), v);
        }
    }
}
template <uint32_t BODY>
__device__ __forceinline__ void store_rows(const TcParams& p, const void* tmC, uint32_t out, int m0, int n0, int lane) {
    constexpr uint32_t CLASS = kBM / 8 * BODY, EDGES = 8 * CLASS;
    constexpr int LAST = BODY / 2;                           // column of the tile's last eight
    const int rows = p.M - m0 < kBM ? p.M - m0 : kBM;
    uint16_t* const c0 = static_cast<uint16_t*>(p.C) + (int64_t)m0 * p.ldc + n0;
    if (lane < 8) tma_store_2d(tmC, out + (uint32_t)lane * CLASS, lane * (int)p.ldc + n0 + (int)rows_head(p, (uint32_t)lane, n0), m0 / 8);
    const uint32_t j = (uint32_t)lane & 7u;
    const bool first0 = j < rows_head(p, (uint32_t)lane >> 3, n0), first1 = j < rows_head(p, ((uint32_t)lane >> 3) + 4u, n0);
#pragma unroll 4
    for (int r = lane >> 3; r < kBM; r += 4) {
        const bool first = (r & 4) ? first1 : first0;
        if (r < rows) c0[(int64_t)r * p.ldc + (first ? 0 : LAST) + j] = lds_u16(out + EDGES + (uint32_t)r * 32u + (first ? 0u : 16u) + 2u * j);
    }
}

// Asks for a bias value without using it.
__device__ __forceinline__ void touch_bias(const TcParams& p, int n) {
    const char* const a = static_cast<const char*>(p.bias) + (int64_t)(n < p.N ? n : p.N - 1) * (p.bias_dtype == BI8_F32 ? 4 : 2);
    asm volatile("{\n\t.reg .u16 v;\n\tld.global.u16 v, [%0];\n\t}" ::"l"(a) : "memory");
}
// The bias of columns n and n + 1, zero outside the output.
__device__ __forceinline__ void bias_pair(const TcParams& p, int n, float& lo, float& hi) {
    lo = n < p.N ? load_as_f32(p.bias, p.bias_dtype, n) : 0.0f;
    hi = n + 1 < p.N ? load_as_f32(p.bias, p.bias_dtype, n + 1) : 0.0f;
}
// The sum of two pairs of a 16-bit type, each rounded once.
__device__ __forceinline__ uint32_t add_pair(uint32_t a, uint32_t b, bool bf) {
    if (bf) {
        const __nv_bfloat162 v = __hadd2_rn(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
        return *reinterpret_cast<const uint32_t*>(&v);
    }
    const __half2 v = __hadd2_rn(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
    return *reinterpret_cast<const uint32_t*>(&v);
}

// Adds residual[m, n] in the output type to a staged row (COLS 16-bit or COLS/2 fp32 values at shared address `row_addr`, columns from
// col0).  Columns and rows outside the output get no addend; they are not stored.
template <int COLS>
__device__ __forceinline__ void add_residual(const TcParams& p, uint32_t row_addr, int m, int col0, bool wide) {
    const bool bf = p.out_dtype == BI8_BF16;
    const int per = wide ? 4 : 8;                       // elements of a 16-byte piece
    const int left = p.N - col0;
    if (m >= p.M) return;
    const int64_t r0 = (int64_t)m * p.ldr + col0;
    if (p.res_vec && COLS / 8 * per <= left) {
        // the row's pieces are all requested before the first is added
        uint4 res[COLS / 8];
#pragma unroll
        for (int g = 0; g < COLS / 8; ++g)
            res[g] = __ldcg(reinterpret_cast<const uint4*>(static_cast<const unsigned char*>(p.residual) + (r0 + g * per) * (wide ? 4 : 2)));
#pragma unroll
        for (int g = 0; g < COLS / 8; ++g) {
            const uint32_t rw[4] = {res[g].x, res[g].y, res[g].z, res[g].w};
            uint32_t w[4];
            lds_v4(row_addr + (uint32_t)(g * 16), w[0], w[1], w[2], w[3]);
#pragma unroll
            for (int u = 0; u < 4; ++u) w[u] = wide ? __float_as_uint(__fadd_rn(__uint_as_float(w[u]), __uint_as_float(rw[u]))) : add_pair(w[u], rw[u], bf);
            sts_v4(row_addr + (uint32_t)(g * 16), w[0], w[1], w[2], w[3]);
        }
    } else {
#pragma unroll 1
        for (int g = 0; g < COLS / 8; ++g)
            add_piece(row_addr + (uint32_t)(g * 16), wide, bf, [&](int e) {
                const int n = g * per + e;
                return n < left ? load_as_f32(p.residual, p.out_dtype, r0 + n) : 0.0f;
            });
    }
}

template <int QB, int MODE, bool SEED, int OUT>
__global__ void __launch_bounds__(Cfg::THREADS, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               const __grid_constant__ CUtensorMap tmSA, const __grid_constant__ CUtensorMap tmSB,
               const __grid_constant__ CUtensorMap tmC, const TcParams p) {
    using C = Cfg;
    using G = Geo<QB>;
    constexpr int BN = C::BN, COLS = C::COLS;
    constexpr bool kScales = (MODE == 0);           // the partial-sum dump uses no scales
    const int store = OUT == kTma16 || OUT == kTma16Add ? kTma : OUT == kRows16 ? kRows : OUT == kOwn16 ? kOwn : p.store;
    const bool wide = OUT == kWide || ((OUT == kAnyOut || OUT == kCluster) && p.out_dtype == BI8_F32);
    const bool addends = OUT != kTma16 && OUT != kRows16 && (OUT == kTma16Add || p.bias != nullptr || p.residual != nullptr);
    extern __shared__ __align__(1024) unsigned char smem_dyn[];
    // dynamic shared memory is only guaranteed 16-byte aligned: round up to the swizzle atom
    const uint32_t raw = smem_u32(smem_dyn);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* base_ptr = smem_dyn + (base - raw);
    const uint32_t bars = base + G::bar_off;
    volatile uint32_t* tmem_holder = reinterpret_cast<volatile uint32_t*>(base_ptr + G::misc_off);
    const uint32_t abort_flag = base + G::misc_off + 4;
    const uint32_t never_flag = base + G::misc_off + 8;
    auto bar = [&](int slot) -> uint32_t { return bars + 8u * (uint32_t)slot; };

    // the warp index through a shuffle: known to be the same in all lanes, so what is derived from it lives in uniform registers
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    const int num_tiles = p.tiles_m * p.tiles_n;
    const int nks = (p.K + kBK - 1) / kBK;
    const int num_items = num_tiles * p.ksplit;
    // limit of the bounded waits in SM cycles: about two seconds, or the diagnostic's shorter one.  The MMA warp's waits
    // get the limit itself and all others four times as much, so that a missing operand stage is reported by the wait
    // that misses it and not by a warp that starves behind it.
    const long long wait_limit_mma = p.wait_limit_us ? (long long)p.wait_limit_us * 2000ll : 4000000000ll;
    const long long wait_limit = p.wait_limit_us ? 4 * wait_limit_mma : wait_limit_mma;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            // the lane that issues the TMA copies; with scales copied by cp.async, every lane of the producer warp as well
            mbar_init(bar(G::FULL_AB + s), (kScales && p.tma_scales != 3) ? 33 : 1);
            mbar_init(bar(G::EMPTY_AB + s), kScales ? 2 : 1);     // the MMAs have read the stage, the seeder its row scales
        }
        for (int b = 0; b < kAccBufs; ++b) {
            mbar_init(bar(G::ACC_FULL + b), kScales ? 2 : 1);     // the block's MMAs and its row records are complete
            mbar_init(bar(G::ACC_EMPTY + b), C::EPI_WARPS);
            mbar_init(bar(G::ACC_SEEDED + b), 1);
        }
        mbar_init(bar(G::OUT_FULL), C::EPI_WARPS);
        mbar_init(bar(G::OUT_EMPTY), 1);
        if (OUT == kCluster)
            for (int w = 0; w < 8; ++w) mbar_init(bar(G::RX_FULL + w), 1);
        sts_u32(abort_flag, 0u);
        sts_u32(never_flag, 0u);                     // a flag nobody raises, for waits that must not be cut short
        mbar_fence_init();
        fence_proxy_async_smem();
        if (OUT == kCluster) {
            // the places of the parts that this CTA finishes: one part from every other CTA
            const int rank = (int)cluster_rank();
            for (int w = rank; w < C::EPI_WARPS; w += p.ksplit) mbar_expect_tx(bar(G::RX_FULL + w / p.ksplit), (uint32_t)(p.ksplit - 1) * G::RX_BYTES);
        }
    }
    if (warp == 1) {
        tmem_alloc(smem_u32((const void*)tmem_holder), 512);
        tmem_relinquish();
    }
    if (SEED) {
        // a row is 2048, 2048, 2048, 0 ... 0: its product with another is 3 * 2^22 = 1.5 * 2^23
        for (uint32_t i = threadIdx.x; i < G::SEED_BYTES / 16; i += C::THREADS)
            sts_v4(base + G::seed_off + i * 16u, (i & 8u) ? 0u : 0x68006800u, (i & 8u) ? 0u : 0x00006800u, 0u, 0u);
        fence_proxy_async_smem();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    if (OUT == kCluster) cluster_arrive();          // the barriers are set up: waited for before the first send
    // Launched so that all of the above may run while the preceding kernel finishes; no global memory is touched before this
    // wait.  The dependents are released by the producer when its last copies are under way: with a small kernel pending from the start (the next
    // quantizer) every block of the K loop was slower (2048 x 4096 x 22016 at block 128 behind a quantizer: 218 us, 199 with the late release).
    wait_predecessor();

    if (warp < kRoleWarps) {
        setmaxnreg_dec<C::ROLE_REGS>();
        if (warp == 0) {
            // ---------------- producer: operand tiles and block scales ----------------
            int stage = 0, sslot = 0;
            uint32_t phase = 0;
            int last_parity[kStages];
#pragma unroll
            for (int s = 0; s < kStages; ++s) last_parity[s] = -1;
            bool ok = true;
            bool first_item = true;
            constexpr uint32_t kSbBytes = (uint32_t)(G::BPS * BN * 4);
            const bool tma_sa = kScales && (p.tma_scales & 1), tma_sb = kScales && (p.tma_scales & 2);
            for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
                int tile, slot, ks0, ks1, m0, n0;
                item_range<OUT>(item, p, nks, tile, slot, ks0, ks1);
                tile_coords<BN>(tile, p, m0, n0);
                for (int ks = ks0; ks < ks1; ++ks) {
                    ok = warp_wait(bar(G::EMPTY_AB + stage), phase ^ 1u, abort_flag, wait_limit);
                    if (!ok) {
                        if (lane == 0) report_timeout(p.status, abort_flag, W_EMPTY_AB);
                        break;
                    }
                    const bool skip = first_item && p.skip_stage >= 0 && ks - ks0 == p.skip_stage;   // diagnostic only
                    const uint32_t fb = bar(G::FULL_AB + stage);
                    const uint32_t sadst = base + G::sa_off + (uint32_t)stage * G::SA_STAGE, sbdst = base + G::sb_off + (uint32_t)sslot * kSbBytes;
                    if (!skip && elect_one()) {
                        mbar_expect_tx(fb, C::STAGE_BYTES + (tma_sa ? G::SA_STAGE : 0u) + (tma_sb ? kSbBytes : 0u));
                        tma_load_2d(base + C::a_off(stage), &tmA, fb, ks * kBK, m0);
                        tma_load_2d(base + C::b_off(stage), &tmB, fb, ks * kBK, n0);
                        // boxes [BPS, 128] and [BPS, BN]; rows and blocks outside the tensors read as zero
                        if (tma_sa) tma_load_2d(sadst, &tmSA, fb, m0, ks * G::BPS);
                        if (tma_sb) tma_load_2d(sbdst, &tmSB, fb, n0, ks * G::BPS);
                    }
                    if (kScales && !(tma_sa && tma_sb) && !skip) {
                        // A scale tensor whose rows are not 16-byte aligned: asynchronous 4-byte copies by the 32 lanes (the
                        // warp does not wait for the data; each lane's arrival on the stage's barrier fires when its
                        // copies have landed)
#pragma unroll
                        for (int blk = 0; blk < G::BPS; ++blk) {
                            const int j = ks * G::BPS + blk;
                            if (!tma_sa) {
                                const float* row = p.sA + (int64_t)j * p.M + m0;
#pragma unroll
                                for (int c = lane; c < kBM; c += 32) {
                                    const bool live = j < p.nb && m0 + c < p.M;
                                    cp_async_4(sadst + (uint32_t)((blk * kBM + c) * 4), live ? row + c : p.sA, live ? 4u : 0u);
                                }
                            }
                            if (!tma_sb) {
                                const float* row = p.sB + (int64_t)j * p.N + n0;
#pragma unroll
                                for (int c = lane; c < BN; c += 32) {
                                    const bool live = j < p.nb && n0 + c < p.N;
                                    cp_async_4(sbdst + (uint32_t)((blk * BN + c) * 4), live ? row + c : p.sB, live ? 4u : 0u);
                                }
                            }
                        }
                        cp_async_arrive(fb);
                    }
                    __syncwarp();
                    if (!skip) {
#pragma unroll
                        for (int s = 0; s < kStages; ++s)
                            if (s == stage) last_parity[s] = (int)phase;
                    }
                    if (++stage == kStages) { stage = 0; phase ^= 1u; }
                    if (++sslot == G::SC_STAGES) sslot = 0;
                }
                first_item = false;
            }
            release_dependents();
            if (!ok) {
                // do not leave while our own copies may still land in this CTA's shared memory
#pragma unroll
                for (int s = 0; s < kStages; ++s)
                    if (last_parity[s] >= 0) (void)mbar_wait(bar(G::FULL_AB + s), (uint32_t)last_parity[s], never_flag, 200000000ll);
            }
        } else if (warp == 1) {
            // ---------------- MMA issuer ----------------
            // Every stage has BPS blocks (blocks past the end of K multiply zero-filled operands) and the blocks go
            // round the three accumulators.  Every tile starts on accumulator 0, so which accumulator a block uses
            // depends only on the stage's position in a cycle of three stages: the K loop runs in such cycles, with the
            // stage body in three copies that have the accumulator as a constant (RotInfo) and no dispatch between
            // them.  The barrier parity of each accumulator flips with every use.
            // One elected thread runs the whole loop: its chain of waits, MMAs and commits per block is what paced the kernel.  As a loop
            // of the warp in which a lane that a comparison picked issued, a block took 640 cycles whatever its width (four columns of
            // promotion work instead of 40 changed nothing); with elect.sync per issue 475, this way 445.
            if (elect_one()) {
                constexpr uint32_t idesc = umma_idesc_i8(kBM, BN);
                int stage = 0;
                uint32_t phase = 0;
                uint32_t accpar[kAccBufs] = {0u, 0u, 0u};
                bool ok = true;
                auto issue_stage = [&](auto rot_tag) {
                    constexpr int ROT = decltype(rot_tag)::value;
                    // a test takes about 80 cycles: those of the stage and of its first accumulator go out together
                    constexpr int buf0 = RotInfo<G::BPS>::buf(ROT, 0), acc_bar = SEED ? G::ACC_SEEDED : G::ACC_EMPTY;
                    const bool full = mbar_test(bar(G::FULL_AB + stage), phase), acc0 = mbar_test(bar(acc_bar + buf0), accpar[buf0]);
                    if (!full) {
                        ok = mbar_wait(bar(G::FULL_AB + stage), phase, abort_flag, wait_limit_mma);
                        if (!ok) {
                            report_timeout(p.status, abort_flag, W_FULL_AB);
                            return;
                        }
                    }
                    const uint64_t adesc = umma_desc_k_sw128(base + C::a_off(stage));
                    const uint64_t bdesc = umma_desc_k_sw128(base + C::b_off(stage));
#pragma unroll
                    for (int blk = 0; blk < G::BPS; ++blk) {
                        const int buf = RotInfo<G::BPS>::buf(ROT, blk);
                        if (blk > 0 || !acc0) ok = mbar_wait(bar(acc_bar + buf), accpar[buf], abort_flag, wait_limit_mma);
                        if (!ok) {
                            report_timeout(p.status, abort_flag, W_ACC_EMPTY);
                            return;
                        }
                        accpar[buf] ^= 1u;
                        tc_fence_after();
#pragma unroll
                        for (int i = 0; i < G::MMAS; ++i) {
                            const uint64_t koff = (uint64_t)((blk * G::MMAS + i) * 32 / 16);
                            mma_i8(tmem_base + (uint32_t)(buf * BN), adesc + koff, bdesc + koff, idesc, (SEED || i > 0) ? 1u : 0u);
                        }
                        tc_commit(bar(G::ACC_FULL + buf));
                    }
                    tc_commit(bar(G::EMPTY_AB + stage));
                    if (++stage == kStages) { stage = 0; phase ^= 1u; }
                };
                for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
                    int tile, slot, ks0, ks1;
                    item_range<OUT>(item, p, nks, tile, slot, ks0, ks1);
                    for (int ks = ks0; ks < ks1 && ok; ks += 3) {
                        issue_stage(std::integral_constant<int, 0>{});
                        if (ks + 1 < ks1 && ok) issue_stage(std::integral_constant<int, 1>{});
                        if (ks + 2 < ks1 && ok) issue_stage(std::integral_constant<int, 2>{});
                    }
                }
            }
            __syncwarp();
        } else if (warp == 2 && (SEED || kScales)) {
            // ---------------- seeder and row records ----------------
            // Follows the accumulators in the order of the MMA issuer, which waits for the seeds' commits instead of the promotion warps;
            // turns a stage's row scales into the records that those read (they wait for both).
            constexpr uint32_t idesc = umma_idesc_f16_f32(kBM, BN);
            const uint64_t desc = umma_desc_k_none(base + G::seed_off, 128, 0);
            int stage = 0;
            uint32_t phase = 0, accpar = 0, rec_off = 0;
            bool ok = true;
            auto seed_acc = [&](int buf) {
                ok = warp_wait(bar(G::ACC_EMPTY + buf), (accpar >> buf) & 1u, abort_flag, wait_limit);
                if (!ok) {
                    if (lane == 0) report_timeout(p.status, abort_flag, W_ACC_EMPTY);
                    return;
                }
                accpar ^= 1u << buf;
                if (SEED) {
                    tc_fence_after();
                    if (elect_one()) {
                        mma_f16_ta(tmem_base + (uint32_t)(buf * BN), tmem_base + (uint32_t)(kAccBufs * BN), desc, idesc, 0u);
                        tc_commit(bar(G::ACC_SEEDED + buf));
                    }
                    __syncwarp();
                }
            };
            int ahead = 0;                    // blocks whose accumulators are seeded already
            for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
                int tile, slot, ks0, ks1;
                item_range<OUT>(item, p, nks, tile, slot, ks0, ks1);
                if (item == (int)blockIdx.x) {
                    // all accumulators are free: seeded while the first operands are on their way
                    const int blocks = (ks1 - ks0) * G::BPS;
                    for (; ahead < kAccBufs && ahead < blocks && ok; ++ahead) seed_acc(ahead);
                }
                int buf = 0;
                for (int ks = ks0; ks < ks1 && ok; ++ks) {
                    if (kScales) {
                        ok = warp_wait(bar(G::FULL_AB + stage), phase, abort_flag, wait_limit);
                        if (!ok) {
                            if (lane == 0) report_timeout(p.status, abort_flag, W_FULL_AB);
                            break;
                        }
#pragma unroll
                        for (int blk = 0; blk < G::BPS; ++blk) {
                            uint32_t v[4], r[8];
                            lds_v4(base + G::sa_off + (uint32_t)stage * G::SA_STAGE + (uint32_t)(blk * kBM * 4 + lane * 16), v[0], v[1], v[2], v[3]);
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                float sxd = __fmul_rn(__uint_as_float(v[u]), 1.0f / (127.0f * 127.0f));
                                if (SEED) sxd = __uint_as_float((__float_as_uint(sxd) + 2u) & 0xFFFFFFFCu);     // 22 significant bits
                                r[2 * u] = __float_as_uint(sxd);
                                r[2 * u + 1] = __float_as_uint(-__fmul_rn(kSeedF, sxd));                         // exact
                            }
                            const uint32_t dst = base + G::row_off + rec_off + (uint32_t)lane * 32u;
                            sts_v4(dst, r[0], r[1], r[2], r[3]);
                            sts_v4(dst + 16u, r[4], r[5], r[6], r[7]);
                            rec_off += G::ROW_REC;
                            if (rec_off == G::ROW_RING) rec_off = 0;
                        }
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar(G::EMPTY_AB + stage));
                        if (++stage == kStages) { stage = 0; phase ^= 1u; }
                    }
#pragma unroll 1
                    for (int blk = 0; blk < G::BPS && ok; ++blk) {
                        if (ahead > 0) --ahead;
                        else seed_acc(buf);
                        if (kScales && ok && lane == 0) mbar_arrive(bar(G::ACC_FULL + buf));
                        if (++buf == kAccBufs) buf = 0;
                    }
                }
            }
        } else if (warp == 3 && MODE == 0 && OUT != kSplit && OUT != kCluster && p.ksplit == 1 && store != kOwn && !wide) {
            // ---------------- storer ----------------
            uint32_t par = 0;
            bool ok = true;
            for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
                int m0, n0;
                tile_coords<BN>(item, p, m0, n0);
                // this wait spans the K loop of a tile: one limit for each of its stages
                ok = false;
                for (int t = 0; t <= nks && !ok; ++t) {
                    ok = warp_wait(bar(G::OUT_FULL), par, abort_flag, wait_limit);
                    if (!ok && __any_sync(0xffffffffu, lds_volatile_u32(abort_flag) != 0u)) break;
                }
                if (!ok) {
                    if (lane == 0) report_timeout(p.status, abort_flag, W_OUT_FULL);
                    break;
                }
                // the promotion warps' writes (ordered by the barrier) before the copies below
                fence_proxy_async_smem();
                // rows and columns of the boxes that lie outside the tensor are not written
                if (OUT == kRows16) {
                    // (a last, partial column of tiles has been stored by the promotion warps)
                    if (n0 + BN <= p.N) store_rows<G::BODY>(p, &tmC, base + G::out_off, m0, n0, lane);
                } else if (lane < C::EPI_WARPS) {
                    const int col0 = n0 + (lane >> 2) * COLS, row0 = m0 + (lane & 3) * 32;
                    if (col0 < p.N && row0 < p.M) tma_store_2d(&tmC, base + G::out_off + (uint32_t)lane * G::PART_BYTES, col0, row0);
                }
                tma_store_commit();
                tma_store_wait_read();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(G::OUT_EMPTY));
                par ^= 1u;
            }
        }
        if (OUT == kCluster) {
            // the cluster's barriers: set-up and, below, teardown (see the promotion warps)
            __syncwarp();
            cluster_wait();
        }
    } else {
        // ---------------- promotion + epilogue ----------------
        setmaxnreg_inc<C::EPI_REGS>();
        const int quarter = warp & 3;                     // tensor-memory lanes 32*quarter .. +31 belong to this warp
        const int slice = (warp - kRoleWarps) >> 2;       // columns COLS*slice .. of the tile
        // A warp reads its 32 x 40 part of an accumulator in two halves of 16 rows, in the shape in which a thread gets the columns 2*c4 and
        // 2*c4 + 1 of every eight and the rows g and g + 8 of each half: rows 8*r + g, r 0 .. 3.  One scale pair then serves four rows.
        const uint32_t g = (uint32_t)lane >> 2, c4 = (uint32_t)lane & 3u;
        const uint32_t t_lane = keep(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(slice * COLS));
        // shared addresses of this thread's first row record and of its first pair of column scales in the rings
        const uint32_t row_addr = keep(base + G::row_off + ((uint32_t)(quarter * 32) + g) * 8u);
        const uint32_t sw_addr = keep(base + G::sb_off + (uint32_t)(slice * COLS * 4) + c4 * 8u);
        const uint32_t bar0 = keep(bars);
        const uint32_t leader = keep(lane == 0 ? 1u : 0u);
        if (SEED && slice == 0) {
            // A of the seeding MMAs: the same rows as B's, in eight spare tensor-memory columns
            static_assert(kAccBufs * BN + 8 <= 512, "no spare tensor-memory columns");
            const uint32_t row_words[8] = {0x68006800u, 0x00006800u, 0u, 0u, 0u, 0u, 0u, 0u};
            tmem_st8(t_lane + (uint32_t)(kAccBufs * BN), row_words);
            tmem_wait_st();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
#pragma unroll
            for (int b = 0; b < kAccBufs; ++b) mbar_arrive(bar(G::ACC_EMPTY + b));
        }
        uint32_t accpar[kAccBufs] = {0u, 0u, 0u};   // barrier parities of the three accumulators, flipped with every use
        uint32_t sc_off = 0, rec_off = 0;         // byte offsets of the block's records in the rings
        bool ok = true;
        uint32_t out_par = 1u;                    // staging area: parity of the release before the tile
        int fail_code = 0;

        // the tile's COLS fp32 accumulators of this thread, kept as packed pairs for fma.rn.f32x2: pair 4*k + r has the columns 8*k + 2*c4, + 1
        // of row 8*r + g
        uint64_t acc2[COLS / 2];
        int m = 0, nbase = 0;                     // first row of the quarter, first column of the slice

        // Promotion of block j, which lies in accumulator `buf_tag`.
        auto promote_block = [&](auto buf_tag, int j) {
            constexpr int buf = decltype(buf_tag)::value;
            const uint32_t t_acc = t_lane + (uint32_t)(buf * BN);
            ok = warp_wait(bar0 + 8u * (uint32_t)(G::ACC_FULL + buf), accpar[buf], abort_flag, wait_limit);
            if (!ok) {
                fail_code = W_ACC_FULL;
                return;
            }
            accpar[buf] ^= 1u;
            tc_fence_after();
            if (MODE == 1) {
#pragma unroll
                for (int c = 0; c < COLS / 8; ++c) {
                    uint32_t pv[8];
                    tmem_ld8(t_acc + (uint32_t)(c * 8), pv);
                    tmem_wait_ld();
                    if (m + lane < p.M && j < p.nb) {
                        int32_t* dst = p.partials + ((int64_t)j * p.M + m + lane) * p.N + nbase + c * 8;
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            if (nbase + c * 8 + i < p.N)
                                dst[i] = SEED ? (int32_t)(pv[i] - kSeedBits) : (int32_t)pv[i];
                    }
                }
                tc_fence_before();
                __syncwarp();
                mbar_arrive_if(bar0 + 8u * (uint32_t)(G::ACC_EMPTY + buf), leader);
            } else {
                // the first eight columns, then the other 32 while those are folded; the accumulator is free when all are in registers
                uint32_t W0[8], W1[4 * COLS / 4 - 8];
                tmem_ld_16x256<8>(t_acc, W0);
                // the rows' records, while the read is in flight
                uint64_t s2[4], n2[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    float sr, nr;
                    lds_pair(row_addr + rec_off + (uint32_t)(r * 64), sr, nr);
                    s2[r] = pack_f32x2(sr, sr);
                    n2[r] = pack_f32x2(nr, nr);
                }
                const uint32_t sw = sw_addr + sc_off;
                tmem_wait_ld();
                tmem_ld_16x256<COLS - 8>(t_acc + 8u, W1);
                fold_columns<SEED, 8, 0, COLS>(W0, sw, s2, n2, acc2);
                tmem_wait_ld();
                tc_fence_before();
                __syncwarp();
                mbar_arrive_if(bar0 + 8u * (uint32_t)(G::ACC_EMPTY + buf), leader);
                fold_columns<SEED, COLS - 8, 8, COLS>(W1, sw, s2, n2, acc2);
                rec_off += G::ROW_REC;
                if (rec_off == G::ROW_RING) rec_off = 0;
                sc_off += G::SC_REC;
                if (sc_off == G::SC_RING) sc_off = 0;
            }
        };

        for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
            int tile, slot, ks0, ks1, m0, n0;
            item_range<OUT>(item, p, nks, tile, slot, ks0, ks1);
            tile_coords<BN>(tile, p, m0, n0);
            m = m0 + quarter * 32;
            nbase = n0 + slice * COLS;
            if (addends && p.bias != nullptr) {
                // into L1, where the epilogue finds it (40 cycles instead of 700)
                touch_bias(p, nbase + lane);
                touch_bias(p, nbase + lane + 32 < nbase + COLS ? nbase + lane + 32 : nbase + lane);
            }
#pragma unroll
            for (int i = 0; i < COLS / 2; ++i) acc2[i] = 0ull;

            // the blocks go round the accumulators; every tile starts on accumulator 0, like the MMA issuer
            const int j1 = ks1 * G::BPS;
#pragma unroll 1
            for (int j = ks0 * G::BPS; j < j1 && ok; j += kAccBufs) {
                promote_block(std::integral_constant<int, 0>{}, j);
                if (j + 1 < j1 && ok) promote_block(std::integral_constant<int, 1>{}, j + 1);
                if (j + 2 < j1 && ok) promote_block(std::integral_constant<int, 2>{}, j + 2);
            }
            bool mine = true;
            if (OUT == kCluster) {
                // The cluster's CTAs hold sums over their shares of K (one tile each; this loop runs once).  Part w of the tile,
                // what warp w of every CTA has, is finished by CTA w mod their number: the others write theirs into its
                // shared memory and it adds them in ascending K order.  (After a wait that ran out a part is sent all the
                // same, so that nobody waits for it.)
                const uint32_t n = (uint32_t)p.ksplit, rank = cluster_rank(), w = (uint32_t)warp - (uint32_t)kRoleWarps;
                const uint32_t owner = w % n, place = base + G::out_off + (w / n) * (n - 1u) * G::RX_BYTES;
                const uint32_t full = bars + 8u * ((uint32_t)G::RX_FULL + w / n);
                mine = owner == rank;
                __syncwarp();
                cluster_wait();
                if (!mine) {
                    // by way of the operand ring: this CTA's MMAs have read their last operands
                    const uint32_t src = base + w * G::RX_BYTES;
#pragma unroll
                    for (int g = 0; g < COLS / 4; ++g) {
                        float v[4];
                        unpack_f32x2(acc2[2 * g], v[0], v[1]);
                        unpack_f32x2(acc2[2 * g + 1], v[2], v[3]);
                        sts_v4(src + (uint32_t)(lane * 16 + g * 512), __float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0)
                        bulk_send(map_to(place + (rank < owner ? rank : rank - 1u) * G::RX_BYTES, owner), src, G::RX_BYTES, map_to(full, owner));
                } else {
                    if (ok) {
                        ok = __all_sync(0xffffffffu, mbar_wait_cluster(full, 0u, abort_flag, wait_limit));
                        if (!ok) fail_code = W_PART;
                    }
                    // Given up, here or before: the others send all the same, at the latest when a wait of theirs runs out, and
                    // neither end of such a copy may be gone before it has landed.
                    if (!ok) (void)mbar_wait_cluster(full, 0u, never_flag, 2 * wait_limit);
#pragma unroll
                    for (int g = 0; g < COLS / 4; ++g) {
                        float own[4], sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                        unpack_f32x2(acc2[2 * g], own[0], own[1]);
                        unpack_f32x2(acc2[2 * g + 1], own[2], own[3]);
#pragma unroll 1
                        for (uint32_t r = 0; r < n; ++r) {
                            uint32_t v[4] = {__float_as_uint(own[0]), __float_as_uint(own[1]), __float_as_uint(own[2]), __float_as_uint(own[3])};
                            if (r != rank) lds_v4(place + (r < rank ? r : r - 1u) * G::RX_BYTES + (uint32_t)(lane * 16 + g * 512), v[0], v[1], v[2], v[3]);
#pragma unroll
                            for (int u = 0; u < 4; ++u) sum[u] = __fadd_rn(sum[u], __uint_as_float(v[u]));
                        }
                        acc2[2 * g] = pack_f32x2(sum[0], sum[1]);
                        acc2[2 * g + 1] = pack_f32x2(sum[2], sum[3]);
                    }
                    __syncwarp();                   // all of the place is read: it may be staged into
                }
            }
            if (!ok) break;
            if (!mine) continue;

            if (MODE == 0 && (OUT == kSplit || (OUT == kAnyOut && slot >= 0))) {
                // Part of a divided tile: straight from the registers to the item's workspace slot, in the order in which
                // the reduction kernel reads it (ws_index: 32 bytes per thread and step, two columns of its four rows).
                float* dst = p.ws + (int64_t)slot * p.slot_floats + ws_index<COLS>(quarter, slice, 0, lane);
                const bool live = quarter * 32 * BN < p.slot_floats;
#pragma unroll
                for (int g = 0; g < COLS / 8; ++g) {
                    if (!live) break;
                    float v[8];
#pragma unroll
                    for (int u = 0; u < 4; ++u) unpack_f32x2(acc2[4 * g + u], v[2 * u], v[2 * u + 1]);
                    stg_v8(dst + g * 256, v);
                }
            } else if (MODE == 0) {
                // The tile leaves through shared memory: the promotion warps write their shares, the storer warp moves them out while
                // the promotion warps go on with the next tile.  Fencing, issuing and waiting for the copies here cost 800 of
                // a K = 512 tile's 7500 cycles (8192 x 512 x 11840: 134 -> 112 us with this and the fast division of tile_coords).  Addresses are derived here from the thread index rather than kept in
                // registers through the K loop, whose register budget is full.  The bias is added to the packed pairs behind the casts (a pair
                // of columns serves four rows), the residual to the staged row.
                uint32_t tid_now;
                asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid_now));
                const uint32_t ln = tid_now & 31u, w = (tid_now >> 5) - (uint32_t)kRoleWarps, qt = w & 3u, sl = w >> 2;
                const uint32_t out = base + G::out_off;
                if (OUT != kCluster && store != kOwn && !wide) {
                    // the copies of the tile before must have read the staging area
                    ok = warp_wait(bar0 + 8u * (uint32_t)G::OUT_EMPTY, out_par, abort_flag, wait_limit);
                    if (!ok) {
                        fail_code = W_OUT_EMPTY;
                        break;
                    }
                    out_par ^= 1u;
                }
                const uint32_t part = OUT == kCluster ? out + (w / (uint32_t)p.ksplit) * ((uint32_t)p.ksplit - 1u) * G::RX_BYTES : out + w * G::PART_BYTES, my_row = part + ln * G::PART_ROW;
                const uint32_t gg = ln >> 2, cc = ln & 3u;
                if (!wide) {
                    const bool bf = p.out_dtype == BI8_BF16;
                    uint32_t e[COLS / 2];
                    if (bf) {
#pragma unroll
                        for (int i = 0; i < COLS / 2; ++i) {
                            float lo, hi;
                            unpack_f32x2(acc2[i], lo, hi);
                            e[i] = pack_bf16x2(lo, hi);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < COLS / 2; ++i) {
                            float lo, hi;
                            unpack_f32x2(acc2[i], lo, hi);
                            e[i] = pack_f16x2(lo, hi);
                        }
                    }
                    if (addends && p.bias != nullptr) {
                        uint32_t b[COLS / 8];
#pragma unroll
                        for (int k = 0; k < COLS / 8; ++k) {
                            float lo, hi;
                            bias_pair(p, nbase + 8 * k + 2 * (int)cc, lo, hi);
                            b[k] = bf ? pack_bf16x2(lo, hi) : pack_f16x2(lo, hi);
                        }
#pragma unroll
                        for (int i = 0; i < COLS / 2; ++i) e[i] = add_pair(e[i], b[i / 4], bf);
                    }
                    const bool own = store == kOwn || (OUT == kRows16 && nbase - (int)sl * COLS + BN > p.N);
                    if (OUT == kRows16 && !own) {
                        // four neighbouring lanes exchange: lane cc gets row 8*cc + gg, all columns
                        uint32_t rowwise[COLS / 2];
#pragma unroll
                        for (int k = 0; k < COLS / 8; ++k) {
                            uint32_t v[4] = {e[4 * k], e[4 * k + 1], e[4 * k + 2], e[4 * k + 3]};
                            transpose4(v, cc);
#pragma unroll
                            for (int u = 0; u < 4; ++u) rowwise[4 * k + u] = v[u];
                        }
                        stage_row<G::BODY>(out + gg * G::CLASS_BYTES + (qt * 4u + cc) * G::BODY, out + G::EDGES + (qt * 32u + 8u * cc + gg) * 32u, sl,
                                           rows_head(p, gg, nbase - (int)sl * COLS), rowwise);
                    } else {
#pragma unroll
                        for (int i = 0; i < COLS / 2; ++i) sts_w(part + (8u * (i & 3) + gg) * G::PART_ROW + (uint32_t)(i / 4) * 16u + cc * 4u, e[i]);
                        if (addends && p.residual != nullptr) {
                            __syncwarp();
                            add_residual<COLS>(p, my_row, m + (int)ln, nbase, wide);
                        }
                    }
                    __syncwarp();
                    if (own) {
                        store_own<(int)G::PART_ROW>(static_cast<unsigned char*>(p.C) + ((int64_t)m * p.ldc + nbase) * 2, p.ldc * 2, part,
                                                    p.M - m, p.N - nbase, wide, (int)ln);
                        __syncwarp();
                    }
                    if (OUT == kCluster) {
                        if (store == kTma) {
                            fence_proxy_async_smem();
                            __syncwarp();
                            if (ln == 0 && nbase < p.N && m < p.M) {
                                tma_store_2d(&tmC, part, nbase, m);
                                tma_store_commit();
                            }
                        }
                    } else if (store != kOwn && ln == 0) {
                        mbar_arrive(bar0 + 8u * (uint32_t)G::OUT_FULL);
                    }
                } else {
                    if (p.bias != nullptr) {
#pragma unroll
                        for (int k = 0; k < COLS / 8; ++k) {
                            float b0, b1;
                            bias_pair(p, nbase + 8 * k + 2 * (int)cc, b0, b1);
#pragma unroll
                            for (int r = 0; r < 4; ++r) {
                                float lo, hi;
                                unpack_f32x2(acc2[4 * k + r], lo, hi);
                                acc2[4 * k + r] = pack_f32x2(__fadd_rn(lo, b0), __fadd_rn(hi, b1));
                            }
                        }
                    }
#pragma unroll 1
                    for (int h = 0; h < 2; ++h) {
                        const int col0 = nbase + h * (COLS / 2), row0 = m;
                        // the previous TMA store must have read the part before it is written again
                        if (store == kTma && ln == 0) tma_store_wait_read();
                        __syncwarp();
                        // groups of eight columns 0 .. 2, then 2 .. 4; the third has columns of both halves
                        static_assert(COLS == 40, "two halves of two and a half groups of eight columns");
#pragma unroll
                        for (int k = 0; k < 3; ++k) {
                            const int c = 8 * k + 2 * (int)cc - 4 * h;
                            if (c >= 0 && c < COLS / 2) {
#pragma unroll
                                for (int r = 0; r < 4; ++r) sts_b64(part + (8u * r + gg) * G::PART_ROW + (uint32_t)c * 4u, acc2[4 * k + r]);
                            }
                        }
                        // the second half finds its groups where the first found its own
#pragma unroll
                        for (int i = 0; i < 12; ++i) acc2[i] = acc2[i + 8];
                        if (p.residual != nullptr) {
                            __syncwarp();
                            add_residual<COLS>(p, my_row, m + (int)ln, col0, wide);
                        }
                        if (store == kTma) {
                            fence_proxy_async_smem();
                            __syncwarp();
                            if (ln == 0 && col0 < p.N && row0 < p.M) {
                                tma_store_2d(&tmC, part, col0, row0);
                                tma_store_commit();
                            }
                        } else {
                            __syncwarp();
                            store_own<(int)G::PART_ROW>(static_cast<unsigned char*>(p.C) + ((int64_t)row0 * p.ldc + col0) * 4, p.ldc * 4, part,
                                                        p.M - row0, p.N - col0, wide, (int)ln);
                            __syncwarp();
                        }
                    }
                }
            }
        }
        // shared memory stays valid until the last store has read it
        if ((wide || OUT == kCluster) && lane == 0) tma_store_wait_read();
        if (!ok) {
            if (lane == 0) report_timeout(p.status, abort_flag, fail_code);
        }
    }

    // ---------------- teardown ----------------
    if (OUT == kCluster) {
        // no CTA leaves while another may still write into its shared memory
        __syncwarp();
        cluster_arrive();
        cluster_wait();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// Reduction of the divided tiles: C[m,n] = cast(sum over the tile's parts) (+ cast(bias[n])) (+ residual[m,n]), the parts added
// in ascending order, so that the result does not depend on scheduling.  A thread adds what one thread of the GEMM has left, one 32-byte
// sector of every part (NP parts in flight: no more registers than the parts need), and stores that: two columns of four rows, a warp 64
// consecutive columns of a row at a time.  (Exchanged between four threads, so that each had eight columns of a row, it was 64-bit shuffles
// and, with eight parts, spills, for wider stores that odd rows could not use.  Layer calls in a graph: 256 x 4096 x 1024 fp32 at block 64, eight
// parts, 15.4 -> 14.2 us, 300 x 3072 x 768 at 32 14.4 -> 14.1, 333 x 1000 x 777 fp16, odd rows of C, 12.5 -> 10.2.)
// The parts come from L2 where they are few (one slot per SM, 12 MB, for outputs of few tiles) and in part from DRAM where they are
// kSplitBytes.  Launched as a programmatic dependent of the GEMM:
// its CTAs are resident as the GEMM's leave.
template <int BN, int COLS, int NP>
__global__ void __launch_bounds__(256) splitk_reduce_kernel(const TcParams p) {
    after_predecessor();
    constexpr int GROUPS = BN / 8;                       // groups of eight columns in a tile row
    const int item = blockIdx.x * 256 + threadIdx.x;
    const int t = item / (kBM * GROUPS), rem = item - t * (kBM * GROUPS);
    const int rb = rem / (GROUPS * 4), x = rem - rb * (GROUPS * 4);
    const int quarter = rb >> 3, g = rb & 7, c = x & 3, cg = x >> 2;
    if (t >= p.tiles_m * p.tiles_n) return;
    int m0, n0;
    tile_coords<BN>(t, p, m0, n0);
    const int m = m0 + quarter * 32 + g, n = n0 + cg * 8 + 2 * c;            // the first of rows 8 apart, the first column
    if (m >= p.M || n >= p.N) return;
    const int slice = cg / (COLS / 8), group = cg - slice * (COLS / 8);
    const float* src = p.ws + (int64_t)t * p.ksplit * p.slot_floats + ws_index<COLS>(quarter, slice, group, 4 * g + c);
    const bool both = n + 1 < p.N, wide = p.out_dtype == BI8_F32, bf = p.out_dtype == BI8_BF16;
    const bool has_bias = p.bias != nullptr, has_res = p.residual != nullptr;
    float b0 = 0.0f, b1 = 0.0f;
    uint32_t res[8];                                     // per row its two values, or one word of two 16-bit ones
    if (has_bias) bias_pair(p, n, b0, b1);
    if (has_res) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int64_t at = (int64_t)(m + 8 * r) * p.ldr + n;
            const bool live = m + 8 * r < p.M;
            res[2 * r] = res[2 * r + 1] = 0u;
            if (wide) {
                const unsigned* const v = static_cast<const unsigned*>(p.residual) + at;
                if (live) res[2 * r] = __ldcg(v);
                if (live && both) res[2 * r + 1] = __ldcg(v + 1);
            } else {
                const unsigned short* const v = static_cast<const unsigned short*>(p.residual) + at;
                if (live && both && p.res_vec) {
                    res[2 * r] = __ldcg(reinterpret_cast<const unsigned*>(v));
                } else if (live) {
                    res[2 * r] = __ldcg(v);
                    if (both) res[2 * r] |= (uint32_t)__ldcg(v + 1) << 16;
                }
            }
        }
    }
    float acc[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) acc[u] = 0.0f;
    for (int s0 = 0; s0 < p.ksplit; s0 += NP) {
        float v[NP][8];
#pragma unroll
        for (int q = 0; q < NP; ++q)
            if (s0 + q < p.ksplit) ldcg_v8(v[q], src + (int64_t)(s0 + q) * p.slot_floats);
#pragma unroll
        for (int q = 0; q < NP; ++q)
            if (s0 + q < p.ksplit) {
#pragma unroll
                for (int u = 0; u < 8; ++u) acc[u] = __fadd_rn(acc[u], v[q][u]);
            }
    }
    const bool vec = both && p.vec_store;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        if (m + 8 * r >= p.M) return;
        const int64_t o = (int64_t)(m + 8 * r) * p.ldc + n;
        float lo = acc[2 * r], hi = acc[2 * r + 1];
        if (wide) {
            if (has_bias) lo = __fadd_rn(lo, b0), hi = __fadd_rn(hi, b1);
            if (has_res) lo = __fadd_rn(lo, __uint_as_float(res[2 * r])), hi = __fadd_rn(hi, __uint_as_float(res[2 * r + 1]));
            float* const d = static_cast<float*>(p.C) + o;
            if (vec) {
                *reinterpret_cast<float2*>(d) = make_float2(lo, hi);
            } else {
                d[0] = lo;
                if (both) d[1] = hi;
            }
        } else {
            uint32_t w = bf ? pack_bf16x2(lo, hi) : pack_f16x2(lo, hi);
            if (has_bias) w = add_pair(w, bf ? pack_bf16x2(b0, b1) : pack_f16x2(b0, b1), bf);
            if (has_res) w = add_pair(w, res[2 * r], bf);
            uint16_t* const d = static_cast<uint16_t*>(p.C) + o;
            if (vec) {
                *reinterpret_cast<uint32_t*>(d) = w;
            } else {
                d[0] = (uint16_t)w;
                if (both) d[1] = (uint16_t)(w >> 16);
            }
        }
    }
}

// Issue-rate probe: back-to-back M128 N256 K32 int8 MMAs on zeroed shared memory, no loads, no epilogue.
__global__ void __launch_bounds__(128, 1) mma_peak_probe_kernel(int iters, int* status) {
    extern __shared__ __align__(1024) unsigned char smem_dyn[];
    const uint32_t raw = smem_u32(smem_dyn);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* base_ptr = smem_dyn + (base - raw);
    __shared__ __align__(8) uint64_t done_bar;
    __shared__ uint32_t holder;
    __shared__ uint32_t abort_word;
    for (uint32_t i = threadIdx.x; i < (kABytes + kProbeN * kBK) / 16; i += blockDim.x)
        reinterpret_cast<uint4*>(base_ptr)[i] = make_uint4(0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u);
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&done_bar), 1);
        abort_word = 0;
        mbar_fence_init();
    }
    fence_proxy_async_smem();
    if (warp == 0) {
        tmem_alloc(smem_u32(&holder), 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *(volatile uint32_t*)&holder;
    if (threadIdx.x == 32) {
        constexpr uint32_t idesc = umma_idesc_i8(kBM, kProbeN);
        const uint64_t adesc = umma_desc_k_sw128(base), bdesc = umma_desc_k_sw128(base + kABytes);
        for (int i = 0; i < iters; ++i) {
            const uint64_t koff = (uint64_t)((i & 3) * 2);
            mma_i8(tmem_base + (uint32_t)((i >> 2) & 1) * kProbeN, adesc + koff, bdesc + koff, idesc, (i >= 8) ? 1u : 0u);
        }
        tc_commit(smem_u32(&done_bar));
        if (!mbar_wait(smem_u32(&done_bar), 0u, smem_u32(&abort_word), 10000000000ll)) report_timeout(status, smem_u32(&abort_word), W_PROBE);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

struct TcMaps {
    CUtensorMap a, b, sa, sb, c;
};

template <int QB, int MODE, bool SEED, int OUT>
int launch_one(const TcMaps& tm, const TcParams& p, int grid, cudaStream_t st) {
    const size_t smem = (OUT == kCluster ? Geo<QB>::cluster_total(p.ksplit) : (size_t)Geo<QB>::total) + 1024;
    static SmemOptIn opt_in;
    const int rc = opt_in.ensure(gemm_tc_kernel<QB, MODE, SEED, OUT>, smem);
    if (rc != BI8_OK) return rc;
    // setmaxnreg.inc waits for registers that the role warps of the same scheduler give up: if the compiler gave the
    // kernel fewer registers per thread than the budget was written for, the wait would never end.  Checked once.
    static int regs_ok = 0;       // 0 unknown, 1 fine, -1 refused
    if (regs_ok == 0) {
        cudaFuncAttributes fa;
        BI8_CUDA_TRY(cudaFuncGetAttributes(&fa, gemm_tc_kernel<QB, MODE, SEED, OUT>));
        regs_ok = ((1 + kPW) * fa.numRegs >= Cfg::ROLE_REGS + kPW * Cfg::EPI_REGS && (1 + kPW) * 32 * fa.numRegs <= 16384) ? 1 : -1;
    }
    if (regs_ok < 0) return fail(BI8_ERR_CUDA, "tensor-core GEMM: the kernel was compiled with a register count its register moves do not fit");
    if (OUT == kCluster) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)grid);
        cfg.blockDim = dim3(Cfg::THREADS);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = (unsigned)p.ksplit;
        attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        BI8_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_tc_kernel<QB, MODE, SEED, OUT>, tm.a, tm.b, tm.sa, tm.sb, tm.c, p));
        return BI8_OK;
    }
    return launch_chained(gemm_tc_kernel<QB, MODE, SEED, OUT>, grid, Cfg::THREADS, smem, st, tm.a, tm.b, tm.sa, tm.sb, tm.c, p);
}

int tc_bn() { return Cfg::BN; }

template <int QB>
int launch_qb(const TcMaps& tm, const TcParams& p, int grid, bool partials, bool seed, bool cluster, cudaStream_t st) {
    if (partials) return seed ? launch_one<QB, 1, true, kAnyOut>(tm, p, grid, st) : launch_one<QB, 1, false, kAnyOut>(tm, p, grid, st);
    if (!seed) return launch_one<QB, 0, false, kAnyOut>(tm, p, grid, st);
    if (cluster) return launch_one<QB, 0, true, kCluster>(tm, p, grid, st);
    if (p.ksplit > 1) return launch_one<QB, 0, true, kSplit>(tm, p, grid, st);
    if (p.out_dtype == BI8_F32) return launch_one<QB, 0, true, kWide>(tm, p, grid, st);
    if constexpr (QB != 32) {
        if (p.store == kRows) return launch_one<QB, 0, true, kRows16>(tm, p, grid, st);
    }
    if (p.store == kOwn) return launch_one<QB, 0, true, kOwn16>(tm, p, grid, st);
    return p.bias || p.residual ? launch_one<QB, 0, true, kTma16Add>(tm, p, grid, st) : launch_one<QB, 0, true, kTma16>(tm, p, grid, st);
}

}  // namespace

// Split-K plan: the K stages of every tile are divided over `ksplit` work items, where that lets the SMs work for a shorter time:
// small outputs that have fewer tiles than the device SMs, and outputs whose tiles fill a last round badly (320 long tiles of a
// weight or input gradient on 148 SMs are three rounds for 2.16 of work).  Partial results go to an fp32 workspace, one slot per
// item, and a second kernel adds them in a fixed order.  (Dividing only the tiles left over after the last full round
// would make equal rows of A give unequal bits, depending on the tile they lie in.)
namespace {
struct SplitPlan {
    int ksplit = 1;
    int stages_per_split = 0;
    int slot_floats = 0;
    size_t bytes = 0;
    bool cluster = false;      // the parts of a tile are the CTAs of a cluster, which add them through shared memory
};
// What a work item takes per stage (128 K-bytes of a tile: four, two or one blocks to promote), what dividing costs whatever its size
// (the second kernel's latency; of its host time a part) and per slot (80 KB written and read again through L2): microseconds.
// Stage: slope over 4 to 32 stages of 4736 undivided tiles, 1.38 us at block 32, 0.68 at 64, 0.43 at 128, of an earlier form of the kernel (8192 x
// 4096 x 11008 now takes 1.22, 0.61 and 0.40 a stage), as is kSplitUs of a reduction that now takes up to a microsecond less.  The parts of a
// tile, and with them the association of its sums, stay as they were; how far the plans are from the best ones of the present
// form is not measured.  The earlier form was checked on a sweep of 1 to 32
// items per tile and clusters of two to four over 23 shapes of 4 to 320 tiles and 6 to 86 stages at the three blocks (GEMM alone in a
// graph): the plan was within 5 % of the best one everywhere and within 2 % in 62 of 69 (block 32 / 64 / 128, the plan's time
// and the undivided one's: 512 x 768 x 768 8.9, 12.0 / 8.0, 8.0 / 6.5, 6.5; 300 x 3072 x 768 12.1, 36.9 / 10.1, 20.4 / 9.3, 13.8; furthest off
// 100 x 2048 x 2048 at 64, 9.4 in four items against 9.0 in six).  The number of items with the lowest sum is taken; the
// largest that the SMs hold is often not the fastest.
double stage_us(int block) { return block <= 32 ? 1.38 : block <= 64 ? 0.68 : 0.43; }
constexpr double kSplitUs = 2.9, kSlotUs = 0.017;
// Where the tiles alone occupy more than half of the SMs, dividing has to save a twentieth, the parts stay below kSplitBytes, and from
// kSplitRounds rounds on nothing is left to be saved.  The parts go to DRAM and back in part (they share 126 MB of L2 with the
// operands) but behind other tiles' loops.  MiB of parts and us, block 64, cold L2: 8192 x 50257 x 768 0 840, 50 724, 75 697, 100 683, 125 677,
// 150 673, 200 704; 768 x 50257 x 8192 0 828, 49 718, 73 683, 97 665, 121 656, 195 659; 4096 x 50257 x 1024 0 568, 52 512, 87 497, 105 515;
// 6144 x 30000 x 1024 0 525, 52 458, 78 447, 105 482; at blocks 32 and 128 the same order.  Beyond the limit 1 to 2 % are left for half as
// much memory again.
constexpr double kSplitWorth = 0.95;
constexpr size_t kSplitBytes = 112u << 20;
constexpr int kSplitRounds = 6;

// The parts of a tile as the CTAs of a cluster: one launch and no workspace, but the exchange, and the later start of a cluster behind a
// kernel that fills the SMs, come to 0.2 + 1.25 us per CTA.  Layer calls, eager / in a graph, against the workspace: 128 x 4096 x
// 11008 in two 22.7 / 24.0 us against 24.5 / 25.4, 300 x 768 x 3072 at block 32 in two 14.3 / 13.5 against 15.9 / 15.6 (undivided),
// 384 x 2048 x 2048 in three 15.3 / 14.4 against 15.8 / 15.0; beyond the line 128 x 4096 x 4096 in four 18.0 / 17.7 against
// 17.3 / 16.6, 256 x 1024 x 1024 in three 11.7 / 10.9 against 11.7 / 10.1.
constexpr double kMeetUs = 0.2, kMeetPartUs = 1.25;
constexpr int kMostCluster = 4;          // what the shared memory has places for
constexpr size_t kSmemLimit = 227 * 1024;
size_t cluster_smem(int block, int n) {
    return 1024 + (block == 32 ? Geo<32>::cluster_total(n) : block == 64 ? Geo<64>::cluster_total(n) : Geo<128>::cluster_total(n));
}
struct ClusterSlots {
    bool known = false;
    int n[kMostCluster + 1] = {0};
};

// `limit`: bytes of workspace that a plan may use.
SplitPlan plan_split(int64_t M, int64_t N, int64_t K, int block, double stage, int sms, const ClusterSlots* slots, size_t limit = SIZE_MAX) {
    SplitPlan pl;
    const int bn = tc_bn();
    const int64_t tiles = ((M + kBM - 1) / kBM) * ((N + bn - 1) / bn);
    const int nks = (int)((K + kBK - 1) / kBK);
    pl.stages_per_split = nks;
    if (tiles <= 0 || nks <= 1 || tiles > kSplitRounds * sms) return pl;
    pl.slot_floats = (int)((M < kBM ? (M + 31) / 32 * 32 : kBM) * bn);
    auto rounds = [&](int64_t items) { return (double)((items + sms - 1) / sms); };
    const bool fills = tiles * 2 > sms;
    double best = rounds(tiles) * stage * nks * (fills ? kSplitWorth : 1.0);
    for (int want = 2; want <= 32 && want <= nks; ++want) {
        const int spp = (nks + want - 1) / want, s = (nks + spp - 1) / spp;
        const size_t bytes = (size_t)tiles * (size_t)s * (size_t)pl.slot_floats * 4;
        if (bytes > limit || (fills ? bytes > kSplitBytes : tiles * want > sms)) break;
        const double cost = rounds(tiles * s) * stage * spp + kSplitUs + kSlotUs * (double)(tiles * s);
        if (cost < best) {
            best = cost;
            pl.ksplit = s;
            pl.stages_per_split = spp;
        }
    }
    // (slots of fewer than 128 rows are smaller than what kSlotUs was measured with; a cluster exchanges whole parts: 40 x 3000 x 5000 takes
    // 14.0 us in four through the workspace and 16.0 in a cluster of four)
    if (pl.ksplit > 1) best -= kSlotUs * (double)(tiles * pl.ksplit) * (1.0 - (double)pl.slot_floats / (kBM * bn));
    for (int c = 2; slots != nullptr && c <= kMostCluster && c <= nks; ++c) {
        const double cost = stage * ((nks + c - 1) / c) + kMeetUs + kMeetPartUs * c;
        if (tiles <= slots->n[c] && cluster_smem(block, c) <= kSmemLimit && cost < best) {
            best = cost;
            pl.ksplit = c;
            pl.stages_per_split = (nks + c - 1) / c;
            pl.cluster = true;
        }
    }
    if (pl.ksplit > 1 && !pl.cluster) pl.bytes = (size_t)tiles * (size_t)pl.ksplit * (size_t)pl.slot_floats * 4;
    return pl;
}

// Clusters of two to kMostCluster CTAs of the general kernel that the device holds at once (asked once per device).
const ClusterSlots* cluster_slots() {
    static ClusterSlots table[64];
    static std::mutex mu;
    int dev = 0;
    if (current_device(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    ClusterSlots& t = table[dev];
    if (!t.known) {
        auto kernel = gemm_tc_kernel<64, 0, true, kCluster>;
        constexpr size_t smem = kSmemLimit;
        static_assert(Geo<32>::total > kSmemLimit / 2 && Geo<64>::total > kSmemLimit / 2 && Geo<128>::total > kSmemLimit / 2, "one CTA per SM at every block size");
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return nullptr;
        const int sms = device_info().sms;
        for (int c = 2; c <= kMostCluster; ++c) {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3((unsigned)(c * (sms / c)));
            cfg.blockDim = dim3(Cfg::THREADS);
            cfg.dynamicSmemBytes = smem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = (unsigned)c;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            if (cudaOccupancyMaxActiveClusters(&t.n[c], kernel, &cfg) != cudaSuccess) {
                (void)cudaGetLastError();
                t.n[c] = 0;
            }
        }
        t.known = true;
    }
    return &t;
}

// The plan of a shape on the current device, with or without clusters, in a workspace of at most `limit` bytes.  A call asks for it two or
// three times (scratch, choice of kernel, launch) at 0.2 to 0.4 us each; each thread keeps the last few (a plan depends on
// nothing but its key).
SplitPlan plan_of(const GemmArgs& g, bool clusters, size_t limit = SIZE_MAX) {
    struct Entry {
        int64_t M = -1, N = 0, K = 0;
        size_t limit = 0;
        int block = 0, dev = 0;
        bool clusters = false;
        SplitPlan plan;
    };
    static thread_local Entry memo[8];
    int dev = 0;
    if (current_device(&dev) != cudaSuccess) dev = 0;
    Entry& e = memo[((uint64_t)(g.M * 31 + g.N * 7 + g.K * 3 + g.block + (int64_t)(limit >> 8) * 5 + (clusters ? 1 : 0)) * 0x9E3779B97F4A7C15ull) >> 61];
    if (e.M != g.M || e.N != g.N || e.K != g.K || e.block != g.block || e.dev != dev || e.clusters != clusters || e.limit != limit) {
        const SplitPlan plan = plan_split(g.M, g.N, g.K, g.block, stage_us(g.block), device_info().sms, clusters ? cluster_slots() : nullptr, limit);
        e.M = g.M;
        e.N = g.N;
        e.K = g.K;
        e.block = g.block;
        e.dev = dev;
        e.clusters = clusters;
        e.limit = limit;
        e.plan = plan;
    }
    return e.plan;
}
}  // namespace

// Whether the undivided tiles occupy more than half of the SMs: a caller without a large workspace does without the split there.
bool gemm_tc_fills_device(const GemmArgs& g) {
    return ((g.M + kBM - 1) / kBM) * ((g.N + tc_bn() - 1) / tc_bn()) * 2 > device_info().sms;
}

size_t gemm_tc_workspace_bytes(const GemmArgs& g, bool used) {
    const DeviceInfo di = device_info();
    if (!di.ok || g.partials != nullptr) return 0;
    return plan_of(g, used).bytes;
}

// Scratch of the division through the workspace at block 64, with the stage time that the refusals of bi8_gemm_dequant_static are
// defined by: which shapes that entry point takes does not move with this kernel's speed.
size_t gemm_tc_static_bytes(int64_t M, int64_t N, int64_t K) {
    const DeviceInfo di = device_info();
    return di.ok ? plan_split(M, N, K, 64, 0.72, di.sms, nullptr).bytes : 0;
}

// For the choice between this kernel and the decode kernel at 33 to 64 rows: a model of this kernel that does not move with its speed (stage
// times of an earlier form, division through the workspace).  What it decides is for which shapes a caller gets the reference's order
// of operations, not only how fast: see gemm_skinny_preferred.
double gemm_tc_estimate_us(const GemmArgs& g) {
    const DeviceInfo di = device_info();
    const double stage = g.block <= 32 ? 1.48 : g.block <= 64 ? 0.72 : 0.45;
    const SplitPlan pl = plan_split(g.M, g.N, g.K, g.block, stage, di.sms, nullptr);
    const int64_t tiles = ((g.M + kBM - 1) / kBM) * ((g.N + tc_bn() - 1) / tc_bn()), items = tiles * pl.ksplit;
    return stage * (double)((items + di.sms - 1) / di.sms * pl.stages_per_split) + 3.5 + (pl.ksplit > 1 ? kSplitUs + kSlotUs * (double)items : 0.0);
}

bool gemm_tc_applicable(const GemmArgs& g, const char** why) {
    auto no = [&](const char* w) {
        if (why) *why = w;
        return false;
    };
    if (g.block != 32 && g.block != 64 && g.block != 128) return no("block size is not 32, 64 or 128");
    if (g.M >= (1ll << 31) - 256 || g.N >= (1ll << 31) - 256 || g.K >= (1ll << 31) - 256) return no("a dimension exceeds 2^31");
    if (!aligned(g.A, 16) || !aligned(g.Bt, 16)) return no("operand base address is not 16-byte aligned");
    if (g.lda % 16 != 0 || g.ldb % 16 != 0) return no("operand row pitch is not a multiple of 16 bytes");
    if (!device_info().ok) return no("device is not compute capability 10.x");
    return true;
}

int launch_gemm_tc(const GemmArgs& g, cudaStream_t st) {
    const DeviceInfo di = device_info();
    if (!di.ok) return fail(BI8_ERR_CUDA, "tensor-core GEMM needs a compute capability 10.x device");
    int dev = 0;
    BI8_CUDA_TRY(current_device(&dev));
    if (dev < 0 || dev >= 64) return fail(BI8_ERR_CUDA, "device ordinal %d out of range", dev);
    const int bps = kBK / g.block;
    const int nb = (int)((g.K + g.block - 1) / g.block);
    TcMaps tm;
    int rc = cached_operand_map(&tm.a, dev, g.A, g.M, g.K, g.lda, kBM);
    if (rc != BI8_OK) return rc;
    const int bn = tc_bn();
    rc = cached_operand_map(&tm.b, dev, g.Bt, g.N, g.K, g.ldb, bn);
    if (rc != BI8_OK) return rc;
    TcParams p{};
    const bool partials = g.partials != nullptr, seed = (g.flags & BI8_GEMM_NO_SEED) == 0;
    // a scale tensor goes through TMA when a tensor map can describe it: 16-byte aligned base and row length
    const bool tma_sa = !partials && aligned(g.sA, 16) && g.M % 4 == 0, tma_sb = !partials && aligned(g.sB, 16) && g.N % 4 == 0;
    p.tma_scales = (tma_sa ? 1 : 0) | (tma_sb ? 2 : 0);
    tm.sa = tm.a;          // stand-ins that are never dereferenced
    tm.sb = tm.b;
    if (tma_sa) {
        rc = cached_scale_map(&tm.sa, dev, g.sA, nb, g.M, kBM, bps);
        if (rc != BI8_OK) return rc;
    }
    if (tma_sb) {
        rc = cached_scale_map(&tm.sb, dev, g.sB, nb, g.N, bn, bps);
        if (rc != BI8_OK) return rc;
    }
    p.sA = g.sA;
    p.sB = g.sB;
    p.bias = g.bias;
    p.C = g.C;
    p.partials = g.partials;
    p.status = device_status_ptr();
    if (!p.status) return BI8_ERR_CUDA;
    p.ldc = g.ldc;
    p.M = (int)g.M;
    p.N = (int)g.N;
    p.K = (int)g.K;
    p.nb = nb;
    p.tiles_m = (int)((g.M + kBM - 1) / kBM);
    p.tiles_n = (int)((g.N + bn - 1) / bn);
    p.out_dtype = g.out_dtype;
    p.bias_dtype = g.bias_dtype;
    const int esz = g.out_dtype == BI8_F32 ? 4 : 2;
    p.vec_store = (g.C != nullptr && aligned(g.C, 16) && (g.ldc * esz) % 16 == 0) ? 1 : 0;
    p.wait_limit_us = g.wait_limit_us;
    p.skip_stage = g.skip_stage;
    tm.c = tm.a;           // stand-in, never dereferenced unless the store mode is kTma
    const int64_t tiles = (int64_t)p.tiles_m * p.tiles_n;
    if (tiles >= (1ll << 31) / 32) return fail(BI8_ERR_SHAPE, "too many output tiles");
    SplitPlan pl;
    pl.stages_per_split = (int)((g.K + kBK - 1) / kBK);
    if (!partials) {
        pl = plan_of(g, seed);
        // the best plan that a smaller workspace has room for (one that is not 16-byte aligned is none): fewer parts, a cluster or no division
        const size_t given = g.workspace != nullptr && aligned(g.workspace, 16) ? g.workspace_bytes : 0;
        if (pl.bytes > given) pl = plan_of(g, seed, given);
    }
    p.ksplit = pl.ksplit;
    p.stages_per_split = pl.stages_per_split;
    p.slot_floats = pl.slot_floats;
    p.residual = g.residual;
    p.ldr = g.ldr;
    p.res_vec = (g.residual != nullptr && aligned(g.residual, 16) && (g.ldr * esz) % 16 == 0) ? 1 : 0;
    p.store = kOwn;
    // (a tensor map clips at 16 bytes: a last piece that is not whole would be written whole)
    if (!partials && (pl.ksplit == 1 || pl.cluster) && p.vec_store && (g.N * esz) % 16 == 0) {
        // one box = what a promotion warp stages per pass: 32 rows x (its columns, or half of them for 4-byte elements)
        const int cols = bn / kPW;
        rc = cached_output_map(&tm.c, dev, g.C, esz, g.M, g.N, g.ldc, 32, esz == 2 ? cols : cols / 2);
        if (rc != BI8_OK) return rc;
        p.store = kTma;
    } else if (!partials && seed && pl.ksplit == 1 && esz == 2 && !g.bias && !g.residual && g.block != 32 && g.M % 8 == 0 && aligned(g.C, 16) &&
               g.ldc < (1ll << 28) && g.N >= bn) {
        // (at block 32 the K loop of that instance is half as long again: 8192 x 4096 x 11005 1835 us, 1230 by own stores, 8192 x 768 x 50257 1670,
        // 1320; at 64 666, 649 and 682, 800; at 128 441, 456 and 531, 611)
        rc = cached_output_map(&tm.c, dev, g.C, 2, g.M / 8, 7 * g.ldc + g.N, 8 * g.ldc, kBM / 8, bn - 8);
        if (rc != BI8_OK) return rc;
        p.store = kRows;
    }
    p.ws = static_cast<float*>(g.workspace);
    p.by_tiles_m = FastDiv(p.tiles_m);
    const int64_t items = tiles * pl.ksplit;
    const int grid = (int)(items < di.sms ? items : di.sms);
    switch (g.block) {
        case 32: rc = launch_qb<32>(tm, p, grid, partials, seed, pl.cluster, st); break;
        case 64: rc = launch_qb<64>(tm, p, grid, partials, seed, pl.cluster, st); break;
        case 128: rc = launch_qb<128>(tm, p, grid, partials, seed, pl.cluster, st); break;
        default: return fail(BI8_ERR_BLOCK, "tensor-core GEMM supports block 32, 64, 128 (got %d)", g.block);
    }
    if (rc != BI8_OK || pl.ksplit == 1 || pl.cluster) return rc;
    constexpr int kTileItems = kBM * (Cfg::BN / 8);
    auto reduce = [&](auto kernel) { return launch_chained(kernel, (unsigned)((tiles * kTileItems + 255) / 256), 256, 0, st, p); };
    constexpr int BN = Cfg::BN, COLS = Cfg::COLS;
    if (pl.ksplit <= 2) return reduce(splitk_reduce_kernel<BN, COLS, 2>);
    return pl.ksplit <= 4 ? reduce(splitk_reduce_kernel<BN, COLS, 4>) : reduce(splitk_reduce_kernel<BN, COLS, 8>);
}

int run_mma_peak_probe(int iters, float* ms, int* sm_count) {
    const DeviceInfo di = device_info();
    if (!di.ok) return fail(BI8_ERR_CUDA, "probe needs a compute capability 10.x device");
    if (iters < 16 || iters > (1 << 22)) return fail(BI8_ERR_LIMIT, "iters must be in [16, 2^22]");
    int* status = device_status_ptr();
    if (!status) return BI8_ERR_CUDA;
    const size_t smem = kABytes + kProbeN * kBK + 1024;
    BI8_CUDA_TRY(cudaFuncSetAttribute(mma_peak_probe_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaEvent_t e0, e1;
    BI8_CUDA_TRY(cudaEventCreate(&e0));
    BI8_CUDA_TRY(cudaEventCreate(&e1));
    mma_peak_probe_kernel<<<di.sms, 128, smem>>>(iters, status);   // warm-up
    BI8_CUDA_TRY(cudaEventRecord(e0));
    mma_peak_probe_kernel<<<di.sms, 128, smem>>>(iters, status);
    BI8_CUDA_TRY(cudaEventRecord(e1));
    BI8_CUDA_TRY(cudaEventSynchronize(e1));
    BI8_CUDA_TRY(cudaEventElapsedTime(ms, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (sm_count) *sm_count = di.sms;
    return BI8_OK;
}

}  // namespace bi8
