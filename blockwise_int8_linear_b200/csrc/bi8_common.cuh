// Shared declarations of the bi8 library's translation units (not part of the public ABI).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <utility>

#include "../../include/bi8.h"

namespace bi8 {

// Records the message returned by bi8_last_error_string() and returns `code`.
int fail(int code, const char* fmt, ...);

// Address of the per-device status word (two ints: code, detail), resolved once per device.
int* device_status_ptr();

inline bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

#define BI8_CUDA_TRY(expr)                                                                    \
    do {                                                                                      \
        cudaError_t e__ = (expr);                                                             \
        if (e__ != cudaSuccess) return ::bi8::fail(BI8_ERR_CUDA, "%s: %s", #expr, cudaGetErrorString(e__)); \
    } while (0)

// The current device, asked for once per call of the C API: an entry point holds a DeviceOfCall while it works (nothing below it changes
// the device), and the launchers, plans and tables that are keyed by device find the answer there.  cudaGetDevice costs 0.1 to
// 0.2 us and a GEMM call asked five times.
struct DeviceOfCall {
    static inline thread_local int depth = 0, dev = -1;
    DeviceOfCall() {
        if (depth++ == 0) dev = -1;
    }
    ~DeviceOfCall() { --depth; }
    DeviceOfCall(const DeviceOfCall&) = delete;
    DeviceOfCall& operator=(const DeviceOfCall&) = delete;
};
inline cudaError_t current_device(int* dev) {
    if (DeviceOfCall::depth > 0 && DeviceOfCall::dev >= 0) {
        *dev = DeviceOfCall::dev;
        return cudaSuccess;
    }
    const cudaError_t e = cudaGetDevice(dev);
    if (e == cudaSuccess && DeviceOfCall::depth > 0) DeviceOfCall::dev = *dev;
    return e;
}

// The opt-in to more than 48 KiB of dynamic shared memory is an attribute of a kernel ON A DEVICE.  A launcher keeps
// one SmemOptIn per kernel instance (a function-local static) and calls ensure() before every launch: the attribute
// is set the first time the instance is used on each device, under a mutex (launchers run on several host threads).
struct SmemOptIn {
    std::mutex mu;
    size_t bytes[64] = {0};
    template <typename Kern>
    int ensure(Kern kern, size_t want) {
        int dev = 0;
        BI8_CUDA_TRY(current_device(&dev));
        if (dev < 0 || dev >= 64) return fail(BI8_ERR_CUDA, "device ordinal %d out of range", dev);
        std::lock_guard<std::mutex> lock(mu);
        if (bytes[dev] >= want) return BI8_OK;
        BI8_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)want));
        bytes[dev] = want;
        return BI8_OK;
    }
};

// Launch that may start before its predecessor in the stream has completed (programmatic stream serialisation).  Every kernel
// launched this way waits for its predecessor (wait_predecessor) in every thread that touches memory which an earlier kernel reads or writes,
// and before it ends, so that "the predecessor has completed" always means that everything before it has completed too.  What a kernel
// reads before its wait is memory that no incomplete earlier kernel writes.  Most kernels release their dependents right after the wait
// (after_predecessor), so that behind them only they themselves are incomplete.  The general GEMM releases later, from its producer warp alone: still
// after the wait, which is for the whole preceding grid.  Two kernels release before their wait: the decode GEMM with early weights, which runs
// only behind this library's own quantizer (that one releases after its wait and writes neither weights nor their scales), and the
// reduction over peers behind such a GEMM, which reads nothing early but its own sequence number.  What follows either may start while two or three
// kernels are incomplete, and waits first thing.  What all this saves is the launch latency and the kernel's set-up, 1-2 us per
// kernel of a chain.
template <typename... P, typename... A>
int launch_chained_grid(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    BI8_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...));
    return BI8_OK;
}

template <typename... P, typename... A>
int launch_chained(void (*kernel)(P...), unsigned grid, unsigned threads, size_t smem, cudaStream_t st, A&&... args) {
    return launch_chained_grid(kernel, dim3(grid), threads, smem, st, std::forward<A>(args)...);
}

#if defined(__CUDACC__)
__device__ __forceinline__ void wait_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void release_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void after_predecessor() {
    wait_predecessor();
    release_dependents();
}
#endif

// Division by a number that the host knows, as a product and a shift: exact for dividends below 2^31.  (A division by a variable is 20
// instructions in 32 bits and 70 to 100 in 64.)
struct FastDiv {
    unsigned mul = 1, d = 1;
    int shift = 0;
    FastDiv() = default;
    explicit FastDiv(int64_t divisor) : d((unsigned)divisor) {
        while ((1ll << shift) < divisor) ++shift;
        mul = (unsigned)((((1ull << shift) - d) << 32) / d + 1);
    }
#if defined(__CUDACC__)
    __device__ __forceinline__ unsigned div(unsigned t) const { return (__umulhi(t, mul) + t) >> shift; }
#endif
};

// ---- launchers implemented in the other translation units -------------------------------------
// (ldq: row pitch of the int8 result in bytes)
int launch_quantize_rowwise(const void* x, int dt, int64_t ldx, int8_t* q, int64_t ldq, float* s, int64_t M, int64_t K,
                            int block, cudaStream_t st);
int launch_quantize_colwise(const void* x, int dt, int64_t ldx, int8_t* q, int64_t ldq, float* s, int64_t R, int64_t C,
                            int block, cudaStream_t st);
// tile quantizer (quantize_tile.cu): column-wise result, and with q_row != nullptr the row-wise result of the same input
bool quantize_tile_applicable(int dt, const void* q_col, int64_t ldqc, const void* q_row, int64_t ldqr, int64_t R, int64_t C, int block);
int launch_quantize_tile(const void* x, int dt, int64_t ldx, int8_t* q_col, int64_t ldqc, float* s_col, int8_t* q_row, int64_t ldqr,
                         float* s_row, int64_t R, int64_t C, int block, cudaStream_t st, float* sums = nullptr);   // sums [ceil(R / 128), C]: column sums of the tile rows (both results only)
constexpr int kTileSumRows = 128;
int launch_column_sum_finish(const float* partial, void* out, int dt, int64_t C, int64_t ranges, cudaStream_t st);
// several small quantizations, column sums and row copies in one launch (quantize.cu)
bool quantize_jobs_fit(const bi8_quantize_task* tasks, int n, int block);
int launch_quantize_jobs(const bi8_quantize_task* tasks, int n, int block, cudaStream_t st);
// sum of the ranks' fp32 partial results over peer memory (peer_reduce.cu)
size_t peer_allreduce_buffer_bytes(int world, int64_t capacity);
int launch_peer_allreduce(void* const* peer_bufs, int rank, int world, int64_t capacity, const float* partial, int64_t M, int64_t N,
                          const void* bias, int bias_dtype, void* out, int out_dtype, unsigned wait_limit_us, cudaStream_t st);
// quantizers with the producing elementwise step in front (quantize_pre.cu)
int launch_quantize_pre(int op, const void* x, const void* x2, int dt, int64_t ldx, const void* weight, float eps, int8_t* q, int64_t ldq,
                        float* sx, int64_t M, int64_t K, int block, cudaStream_t st);
// C[m, n] += R[m, n] in the type of C (C may be R)
int launch_residual_add(void* C, int64_t ldc, const void* R, int64_t ldr, int dt, int64_t M, int64_t N, cudaStream_t st);
// prefill-sized sum over ranks: reduce-scatter by peer loads, all-gather by peer stores (peer_reduce_large.cu)
size_t peer_allreduce_large_buffer_bytes(int64_t capacity);
size_t peer_allreduce_large_partial_offset();
size_t peer_allreduce_large_out_offset(int64_t capacity);
int launch_peer_allreduce_large(void* const* peer_bufs, int rank, int world, int64_t capacity, int64_t M, int64_t N, const void* bias,
                                int bias_dtype, int out_dtype, unsigned wait_limit_us, cudaStream_t st);
// rotary embedding of q and k and the append of k and v to the caches for one decode step (rope_cache.cu)
int launch_rope_cache_append(const void* qkv, int dt, const float* cis, const long long* pos, void* q_out, void* kcache, void* vcache,
                             int64_t B, int64_t H, int64_t D, int64_t max_len, cudaStream_t st);
// int8 rows of any alignment to rows on 16-byte boundaries (copy_rows.cu)
int launch_copy_rows(const int8_t* src, int64_t lds, int8_t* dst, int64_t ldd, int64_t rows, int64_t cols, cudaStream_t st);
// column sums in fp32 (column_sum.cu)
size_t column_sum_workspace_bytes(int64_t R, int64_t C);
int launch_column_sum(const void* x, int dt, int64_t ldx, void* out, int64_t R, int64_t C, void* workspace, size_t workspace_bytes,
                      cudaStream_t st);
int launch_dequantize_rowwise(const int8_t* q, int64_t ldq, const float* s, void* out, int dt, int64_t M, int64_t K,
                              int block, cudaStream_t st);

// Row-parallel layers: the fp32 result in C is this rank's partial result, which a kernel launched behind the decode GEMM (resident
// as it ends) exchanges over peer memory (peer_common.cuh).
struct PeerEpilogue {
    const void* args;         // const PeerArgs*
    const void* bias;
    int bias_dtype;
    void* out;                // [M, N] of out_dtype, contiguous
    int out_dtype;
    long long limit_cycles;
};

struct GemmArgs {
    const int8_t* A;
    int64_t lda;
    const int8_t* Bt;
    int64_t ldb;
    const float* sA;
    const float* sB;
    const void* bias;
    int bias_dtype;
    void* C;
    int64_t ldc;
    int out_dtype;
    int32_t* partials;  // non-null: write int32 block partial sums [nb, M, N] instead of C
    int64_t M, N, K;
    int block;
    int flags;
    void* workspace;          // optional scratch for split-K partial results
    size_t workspace_bytes;
    const void* X = nullptr;  // decode kernel, non-null: activations before quantization (A and sA unused), quantized inside it
    int x_dtype = 0;
    int64_t ldx = 0;
    int pre_op = BI8_PRE_NONE;          // ... with this step in front: X2 is the second operand of SiLU * mul (same pitch) or the RMSNorm weight
    const void* X2 = nullptr;
    float eps = 0.0f;
    bool after_own_quantizer = false;   // the kernel launched just before is this library's decode quantizer
    unsigned wait_limit_us = 0;         // diagnostic: limit of the general kernel's bounded waits (0 = default, about 2 s)
    int skip_stage = -1;                // diagnostic: the general kernel's producer leaves this stage of its first item out
    const PeerEpilogue* peer = nullptr; // decode kernel only: sum C over the ranks in a kernel behind it
    const void* residual = nullptr;     // general tensor-core kernel only: [M, N] addend of the output type, added after the bias
    int64_t ldr = 0;                    // its row pitch in elements
    int64_t bias_ld = 0;                // decode kernel only: row pitch of `bias` in elements; non-zero makes it an [M, N] addend
};

bool gemm_tc_applicable(const GemmArgs& g, const char** why);
size_t gemm_tc_workspace_bytes(const GemmArgs& g, bool used);   // `used`: nothing where clusters add the parts
size_t gemm_tc_static_bytes(int64_t M, int64_t N, int64_t K);
bool gemm_tc_fills_device(const GemmArgs& g);
int launch_gemm_tc(const GemmArgs& g, cudaStream_t st);
int launch_gemm_generic(const GemmArgs& g, cudaStream_t st);
double gemm_tc_estimate_us(const GemmArgs& g);       // few tiles: the time the general kernel takes, for a choice between kernels
bool gemm_skinny_applicable(const GemmArgs& g);
int64_t gemm_skinny_part(const GemmArgs& g);
bool gemm_skinny_preferred(const GemmArgs& g);
int launch_gemm_skinny(const GemmArgs& g, cudaStream_t st);
int launch_skinny_quantize(const void* x, int x_dtype, int64_t ldx, int8_t* q, float* sx, int64_t M, int64_t K, int block,
                           cudaStream_t st);
bool gemm_smallm_applicable(const GemmArgs& g);
int launch_gemm_smallm(const GemmArgs& g, cudaStream_t st);
int run_mma_peak_probe(int iters, float* ms, int* sm_count);

// ---- small device helpers ----------------------------------------------------------------------
__device__ __forceinline__ uint4 ld_nc_v4(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

__device__ __forceinline__ float bf16lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// fp32 -> bf16 bits, round to nearest even (two values packed: lo in bits 0-15)
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

}  // namespace bi8
