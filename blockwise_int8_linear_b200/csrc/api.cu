// extern "C" surface of libbi8.so: argument validation, dispatch, error text.  See include/bi8.h.
#include "bi8_common.cuh"
#include "peer_common.cuh"

#include <cstdarg>
#include <cstdio>
#include <mutex>

namespace bi8 {

namespace {
thread_local char g_err[512] = "";

// Per-device status word of the kernels' bounded waits: {code, detail}.
__device__ int g_status[2];
}  // namespace

int fail(int code, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}

int* device_status_ptr() {
    static int* ptrs[64] = {nullptr};
    static std::mutex mu;
    int dev = 0;
    if (current_device(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        fail(BI8_ERR_CUDA, "cudaGetDevice failed");
        return nullptr;
    }
    std::lock_guard<std::mutex> lock(mu);
    if (!ptrs[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_status);
        if (e != cudaSuccess) {
            fail(BI8_ERR_CUDA, "cudaGetSymbolAddress(status): %s", cudaGetErrorString(e));
            return nullptr;
        }
        ptrs[dev] = static_cast<int*>(p);
    }
    return ptrs[dev];
}

namespace {

bool dtype_ok(int dt) { return dt == BI8_BF16 || dt == BI8_F32 || dt == BI8_F16; }
int dtype_size(int dt) { return dt == BI8_F32 ? 4 : 2; }

// `quantized`: the activations are there as int8 (A, sA); false where the GEMM kernel may quantize them itself.
int check_gemm(const GemmArgs& g, bool partials, bool quantized = true) {
    if (g.M < 0 || g.N < 0 || g.K < 0) return fail(BI8_ERR_SHAPE, "gemm: negative dimension (M=%lld N=%lld K=%lld)", (long long)g.M, (long long)g.N, (long long)g.K);
    if (g.block < 1) return fail(BI8_ERR_BLOCK, "gemm: block size %d", g.block);
    if (g.M == 0 || g.N == 0) return BI8_OK;
    if (g.K > 0 && ((quantized && !g.A) || !g.Bt)) return fail(BI8_ERR_NULL, "gemm: null operand");
    if (g.lda < g.K || g.ldb < g.K) return fail(BI8_ERR_SHAPE, "gemm: row pitch smaller than K");
    if (partials) {
        if (!g.partials && g.K > 0) return fail(BI8_ERR_NULL, "gemm_block_partials: null output");
    } else {
        if (!g.C) return fail(BI8_ERR_NULL, "gemm: null output");
        if (g.K > 0 && ((quantized && !g.sA) || !g.sB)) return fail(BI8_ERR_NULL, "gemm: null scale tensor");
        if (!dtype_ok(g.out_dtype)) return fail(BI8_ERR_DTYPE, "gemm: unknown output dtype code %d", g.out_dtype);
        if (g.bias && !dtype_ok(g.bias_dtype)) return fail(BI8_ERR_DTYPE, "gemm: unknown bias dtype code %d", g.bias_dtype);
        if (g.ldc < g.N) return fail(BI8_ERR_SHAPE, "gemm: ldc smaller than N");
        if (!aligned(g.C, dtype_size(g.out_dtype))) return fail(BI8_ERR_ALIGN, "gemm: output not element aligned");
    }
    return BI8_OK;
}

// Whether the memory of the residual [M, N] (row pitch ldr) and of the output meet anywhere between their first and last elements.
bool overlaps_output(const void* residual, int64_t ldr, const void* C, int64_t ldc, int out_dtype, int64_t M, int64_t N) {
    if (residual == nullptr || C == nullptr || M <= 0 || N <= 0) return false;
    const int esz = dtype_size(out_dtype);
    const char *c0 = static_cast<const char*>(C), *c1 = c0 + ((M - 1) * ldc + N) * esz;
    const char *r0 = static_cast<const char*>(residual), *r1 = r0 + ((M - 1) * ldr + N) * esz;
    return r0 < c1 && c0 < r1;
}

// The kernels that do not add GemmArgs::residual themselves are followed by one that does.
int then_residual(int rc, const GemmArgs& g, cudaStream_t st) {
    if (rc != BI8_OK || g.residual == nullptr) return rc;
    return launch_residual_add(g.C, g.ldc, g.residual, g.ldr, g.out_dtype, g.M, g.N, st);
}

int dispatch_gemm(const GemmArgs& g, cudaStream_t st) {
    const char* why = "";
    const bool tc_ok = g.K > 0 && gemm_tc_applicable(g, &why);
    if (g.flags & BI8_GEMM_FORCE_SMALLM) {
        if (!gemm_smallm_applicable(g)) return fail(BI8_ERR_ALIGN, "small-M GEMM not applicable (needs M <= 16, block 32/64/128, K %% 16 == 0, 32-byte aligned weight rows)");
        return then_residual(launch_gemm_smallm(g, st), g, st);
    }
    if (g.flags & BI8_GEMM_FORCE_SKINNY) {
        if (!gemm_skinny_applicable(g))
            return fail(BI8_ERR_ALIGN, "skinny tensor-core GEMM not applicable (needs M <= 64, block 32/64/128, N %% 4 == 0, 16-byte aligned "
                                       "operand rows and weight scales)");
        return then_residual(launch_gemm_skinny(g, st), g, st);
    }
    const bool free_choice = !(g.flags & (BI8_GEMM_FORCE_TC | BI8_GEMM_FORCE_GENERIC)) && g.K > 0;
    // M <= 64: one pass over the weights on the tensor cores with exchanged operand roles
    if (free_choice && gemm_skinny_preferred(g)) return then_residual(launch_gemm_skinny(g, st), g, st);
    // otherwise M <= 8 streams the weights on the CUDA cores; 9..16 would stream them twice and is faster on the
    // general tensor-core kernel
    if (free_choice && g.M <= 8 && gemm_smallm_applicable(g)) return then_residual(launch_gemm_smallm(g, st), g, st);
    if (g.flags & BI8_GEMM_FORCE_TC) {
        if (!tc_ok) return fail(BI8_ERR_ALIGN, "tensor-core GEMM not applicable: %s", why);
        return launch_gemm_tc(g, st);
    }
    if ((g.flags & BI8_GEMM_FORCE_GENERIC) || !tc_ok || g.K == 0) return then_residual(launch_gemm_generic(g, st), g, st);
    return launch_gemm_tc(g, st);
}

// Where a decode-sized layer quantizes its activations: inside the GEMM (one launch; every cluster repeats the work and the weights
// wait for the predecessor) or in a kernel in front of it (weights and quantizer overlap).  In a chain of steps inside up to
// this many values: 3 x 2048: 37 us a layer against 47, 1 x 4096: 61 against 65, but 8 x 4096: 78 against 71.  A plain call by itself
// is bound by its launches as long as a CTA's part is no longer than that: inside against in front, 16 x 4096 -> 4096 (16384
// values a CTA) 11.4 us, 13.9; 8 x 4096 -> 11008 (32768) 19.4, 15.6; 16 x 5120 -> 13824 (81920) 33, 20.
constexpr int64_t kQuantInKernelValues = BI8_ONE_LAUNCH_VALUES;

// Decode-sized layer (the weight-streaming GEMM and what produces its activations).  `g` describes the GEMM on the
// quantized activations g.A / g.sA, which are scratch (null: none); `alone`: a plain call, not a step with a producer or a
// residual around it.  Sets *done to false, having launched nothing, where
// that kernel does not take the shape.
int launch_decode(GemmArgs g, bool alone, int op, const void* x, const void* x2, const void* norm_weight, int x_dtype, int64_t ldx, float eps, bool* done,
                  cudaStream_t st) {
    *done = true;
    GemmArgs in = g;
    in.X = x;
    in.x_dtype = x_dtype;
    in.ldx = ldx;
    in.pre_op = op;
    in.X2 = op == BI8_PRE_SILU_MUL ? x2 : op == BI8_PRE_RMSNORM ? norm_weight : nullptr;
    in.eps = eps;
    const bool scratch = g.A != nullptr && g.sA != nullptr;
    const bool forced_in = (g.flags & BI8_GEMM_QUANT_IN_KERNEL) || !scratch;
    const bool want_in = forced_in || (g.M <= 16 && (g.M * g.K <= kQuantInKernelValues || (alone && gemm_skinny_part(in) <= kQuantInKernelValues)));
    if (want_in && !(op == BI8_PRE_SILU_MUL && !x2) && gemm_skinny_applicable(in)) return launch_gemm_skinny(in, st);
    if (!scratch || g.K % 16 != 0 || !aligned(g.A, 16) || !gemm_skinny_preferred(g)) {
        *done = false;
        return BI8_OK;
    }
    // a quantizer in front; none of this library's writes weights, so the GEMM's set-up and first weight copies overlap it, and
    // it waits for the quantizer's completion before it reads the activations
    const bool vec = aligned(x, 16) && (ldx * dtype_size(x_dtype)) % 16 == 0 && g.K % 8 == 0;    // 8 elements per load
    int8_t* xq = const_cast<int8_t*>(g.A);
    float* sx = const_cast<float*>(g.sA);
    const int rc = op == BI8_PRE_NONE && vec ? launch_skinny_quantize(x, x_dtype, ldx, xq, sx, g.M, g.K, g.block, st)
                                             : launch_quantize_pre(op, x, x2, x_dtype, ldx, norm_weight, eps, xq, g.K, sx, g.M, g.K, g.block, st);
    if (rc != BI8_OK) return rc;
    g.after_own_quantizer = true;
    return launch_gemm_skinny(g, st);
}

}  // namespace
}  // namespace bi8

using namespace bi8;

extern "C" {

int bi8_version(void) { return BI8_VERSION; }

const char* bi8_last_error_string(void) { return g_err; }

int bi8_device_status(int* detail) {
    int* p = device_status_ptr();
    if (!p) return BI8_ERR_CUDA;
    int host[2] = {0, 0};
    BI8_CUDA_TRY(cudaDeviceSynchronize());
    BI8_CUDA_TRY(cudaMemcpy(host, p, sizeof(host), cudaMemcpyDeviceToHost));
    if (host[0] != 0) {
        int zero[2] = {0, 0};
        BI8_CUDA_TRY(cudaMemcpy(p, zero, sizeof(zero), cudaMemcpyHostToDevice));
        if (detail) *detail = host[1];
        return fail(host[0], "a device-side bounded wait gave up (wait code %d)", host[1]);
    }
    if (detail) *detail = 0;
    return BI8_OK;
}

int bi8_quantize_rowwise_pitched(const void* x, int x_dtype, int64_t ldx, int8_t* q, int64_t ldq, float* s, int64_t M, int64_t K, int block,
                                 void* stream) {
    DeviceOfCall call;
    if (!dtype_ok(x_dtype)) return fail(BI8_ERR_DTYPE, "quantize_rowwise: unknown dtype code %d", x_dtype);
    if (block < 1) return fail(BI8_ERR_BLOCK, "quantize_rowwise: block size %d", block);
    if (M < 0 || K < 0 || ldx < K || ldq < K) return fail(BI8_ERR_SHAPE, "quantize_rowwise: bad shape M=%lld K=%lld ldx=%lld ldq=%lld", (long long)M, (long long)K, (long long)ldx, (long long)ldq);
    if (M == 0 || K == 0) return BI8_OK;
    if (!x || !q || !s) return fail(BI8_ERR_NULL, "quantize_rowwise: null pointer");
    if (!aligned(x, dtype_size(x_dtype)) || !aligned(s, 4)) return fail(BI8_ERR_ALIGN, "quantize_rowwise: pointer not element aligned");
    return launch_quantize_rowwise(x, x_dtype, ldx, q, ldq, s, M, K, block, static_cast<cudaStream_t>(stream));
}

int bi8_quantize_rowwise(const void* x, int x_dtype, int64_t ldx, int8_t* q, float* s, int64_t M, int64_t K, int block,
                         void* stream) {
    return bi8_quantize_rowwise_pitched(x, x_dtype, ldx, q, K, s, M, K, block, stream);
}

int bi8_quantize_colwise_pitched(const void* x, int x_dtype, int64_t ldx, int8_t* q, int64_t ldq, float* s, int64_t R, int64_t C, int block,
                                 void* stream) {
    DeviceOfCall call;
    if (!dtype_ok(x_dtype)) return fail(BI8_ERR_DTYPE, "quantize_colwise: unknown dtype code %d", x_dtype);
    if (block < 1) return fail(BI8_ERR_BLOCK, "quantize_colwise: block size %d", block);
    if (R < 0 || C < 0 || ldx < C || ldq < R) return fail(BI8_ERR_SHAPE, "quantize_colwise: bad shape R=%lld C=%lld ldx=%lld ldq=%lld", (long long)R, (long long)C, (long long)ldx, (long long)ldq);
    if (R == 0 || C == 0) return BI8_OK;
    if (!x || !q || !s) return fail(BI8_ERR_NULL, "quantize_colwise: null pointer");
    if (!aligned(x, dtype_size(x_dtype)) || !aligned(s, 4)) return fail(BI8_ERR_ALIGN, "quantize_colwise: pointer not element aligned");
    return launch_quantize_colwise(x, x_dtype, ldx, q, ldq, s, R, C, block, static_cast<cudaStream_t>(stream));
}

int bi8_quantize_colwise(const void* x, int x_dtype, int64_t ldx, int8_t* q, float* s, int64_t R, int64_t C, int block,
                         void* stream) {
    return bi8_quantize_colwise_pitched(x, x_dtype, ldx, q, R, s, R, C, block, stream);
}

int bi8_quantize_dual_pitched(const void* x, int x_dtype, int64_t ldx, int8_t* q_row, int64_t ldq_row, float* s_row, int8_t* q_col, int64_t ldq_col,
                              float* s_col, int64_t R, int64_t C, int block, void* stream) {
    DeviceOfCall call;
    if (!dtype_ok(x_dtype)) return fail(BI8_ERR_DTYPE, "quantize_dual: unknown dtype code %d", x_dtype);
    if (block < 1) return fail(BI8_ERR_BLOCK, "quantize_dual: block size %d", block);
    if (R < 0 || C < 0 || ldx < C || ldq_row < C || ldq_col < R)
        return fail(BI8_ERR_SHAPE, "quantize_dual: bad shape R=%lld C=%lld ldx=%lld ldq=%lld, %lld", (long long)R, (long long)C, (long long)ldx, (long long)ldq_row, (long long)ldq_col);
    if (R == 0 || C == 0) return BI8_OK;
    if (!x || !q_row || !s_row || !q_col || !s_col) return fail(BI8_ERR_NULL, "quantize_dual: null pointer");
    if (!aligned(x, dtype_size(x_dtype)) || !aligned(s_row, 4) || !aligned(s_col, 4)) return fail(BI8_ERR_ALIGN, "quantize_dual: pointer not element aligned");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (quantize_tile_applicable(x_dtype, q_col, ldq_col, q_row, ldq_row, R, C, block))
        return launch_quantize_tile(x, x_dtype, ldx, q_col, ldq_col, s_col, q_row, ldq_row, s_row, R, C, block, st);
    // what the one-pass kernel does not take: the two single-purpose quantizers, same results
    const int rc = launch_quantize_rowwise(x, x_dtype, ldx, q_row, ldq_row, s_row, R, C, block, st);
    if (rc != BI8_OK) return rc;
    return launch_quantize_colwise(x, x_dtype, ldx, q_col, ldq_col, s_col, R, C, block, st);
}

size_t bi8_quantize_dual_sum_workspace_bytes(int x_dtype, int64_t R, int64_t C, int block) {
    if (x_dtype == BI8_F32 || !dtype_ok(x_dtype) || R < 0 || C < 0 || R >= (1ll << 31) - 256 || C >= (1ll << 31) - 65536) return 0;
    if (block != 32 && block != 64 && block != 128) return 0;
    return (size_t)((R + kTileSumRows - 1) / kTileSumRows) * (size_t)C * 4;
}

int bi8_quantize_dual_sum(const void* x, int x_dtype, int64_t ldx, int8_t* q_row, int64_t ldq_row, float* s_row, int8_t* q_col, int64_t ldq_col,
                          float* s_col, void* sum, int64_t R, int64_t C, int block, void* workspace, size_t workspace_bytes, void* stream) {
    DeviceOfCall call;
    if (R <= 0 || C <= 0 || ldx < C || ldq_row < C || ldq_col < R) return fail(BI8_ERR_SHAPE, "quantize_dual_sum: bad shape R=%lld C=%lld ldx=%lld", (long long)R, (long long)C, (long long)ldx);
    const size_t need = bi8_quantize_dual_sum_workspace_bytes(x_dtype, R, C, block);
    if (need == 0) return fail(BI8_ERR_LIMIT, "quantize_dual_sum: 16-bit inputs and blocks of 32, 64 or 128");
    if (!x || !q_row || !s_row || !q_col || !s_col || !sum) return fail(BI8_ERR_NULL, "quantize_dual_sum: null pointer");
    if (!workspace || workspace_bytes < need || !aligned(workspace, 4)) return fail(BI8_ERR_WORKSPACE, "quantize_dual_sum: workspace missing or too small");
    if (!aligned(x, 2) || !aligned(sum, 2) || !aligned(s_row, 4) || !aligned(s_col, 4)) return fail(BI8_ERR_ALIGN, "quantize_dual_sum: pointer not element aligned");
    if (!quantize_tile_applicable(x_dtype, q_col, ldq_col, q_row, ldq_row, R, C, block))
        return fail(BI8_ERR_ALIGN, "quantize_dual_sum: int8 rows do not begin on 16-byte boundaries");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    float* partial = static_cast<float*>(workspace);
    const int rc = launch_quantize_tile(x, x_dtype, ldx, q_col, ldq_col, s_col, q_row, ldq_row, s_row, R, C, block, st, partial);
    return rc != BI8_OK ? rc : launch_column_sum_finish(partial, sum, x_dtype, C, (R + kTileSumRows - 1) / kTileSumRows, st);
}

int bi8_quantize_dual(const void* x, int x_dtype, int64_t ldx, int8_t* q_row, float* s_row, int8_t* q_col, float* s_col, int64_t R,
                      int64_t C, int block, void* stream) {
    return bi8_quantize_dual_pitched(x, x_dtype, ldx, q_row, C, s_row, q_col, R, s_col, R, C, block, stream);
}

int bi8_quantize_many_fits(const bi8_quantize_task* tasks, int n, int block) {
    return tasks && n > 0 && quantize_jobs_fit(tasks, n, block) ? 1 : 0;
}

int bi8_quantize_many(const bi8_quantize_task* tasks, int n, int block, void* stream) {
    DeviceOfCall call;
    if (n < 0 || (n > 0 && !tasks)) return fail(BI8_ERR_NULL, "quantize_many: null pointer");
    if (block < 1) return fail(BI8_ERR_BLOCK, "quantize_many: block size %d", block);
    const bool fits = n > 0 && quantize_jobs_fit(tasks, n, block);
    for (int i = 0; i < n; ++i) {
        const bi8_quantize_task& t = tasks[i];
        const bool copy = t.x_dtype == BI8_I8;
        if (!copy && !dtype_ok(t.x_dtype)) return fail(BI8_ERR_DTYPE, "quantize_many: unknown dtype code %d", t.x_dtype);
        if (t.rows < 0 || t.cols < 0 || t.ldx < t.cols || (t.q_row && t.ldq_row < t.cols) || (t.q_col && t.ldq_col < t.rows))
            return fail(BI8_ERR_SHAPE, "quantize_many: bad shape of task %d", i);
        if (copy && (!t.q_row || !aligned(t.q_row, 16) || t.ldq_row % 16 != 0 || t.ldq_row < (t.cols + 15) / 16 * 16))
            return fail(BI8_ERR_ALIGN, "quantize_many: rows of task %d do not begin on 16-byte boundaries", i);
        if (t.rows == 0 || t.cols == 0) continue;
        if (!t.x || (!copy && ((t.q_row && !t.s_row) || (t.q_col && !t.s_col)))) return fail(BI8_ERR_NULL, "quantize_many: null pointer in task %d", i);
        if (!copy && (!aligned(t.x, dtype_size(t.x_dtype)) || (t.q_row && !aligned(t.s_row, 4)) || (t.q_col && !aligned(t.s_col, 4)) ||
                      (t.sum && !aligned(t.sum, dtype_size(t.x_dtype)))))
            return fail(BI8_ERR_ALIGN, "quantize_many: pointer of task %d not element aligned", i);
        if (t.sum && !fits) return fail(BI8_ERR_LIMIT, "quantize_many: column sums only where the tasks fit one launch");
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (fits) return launch_quantize_jobs(tasks, n, block, st);
    for (int i = 0; i < n; ++i) {
        const bi8_quantize_task& t = tasks[i];
        int rc = BI8_OK;
        if (t.x_dtype == BI8_I8) rc = bi8_copy_rows(static_cast<const int8_t*>(t.x), t.ldx, t.q_row, t.ldq_row, t.rows, t.cols, stream);
        else if (t.q_row && t.q_col)
            rc = bi8_quantize_dual_pitched(t.x, t.x_dtype, t.ldx, t.q_row, t.ldq_row, t.s_row, t.q_col, t.ldq_col, t.s_col, t.rows, t.cols, block, stream);
        else if (t.q_row) rc = bi8_quantize_rowwise_pitched(t.x, t.x_dtype, t.ldx, t.q_row, t.ldq_row, t.s_row, t.rows, t.cols, block, stream);
        else if (t.q_col) rc = bi8_quantize_colwise_pitched(t.x, t.x_dtype, t.ldx, t.q_col, t.ldq_col, t.s_col, t.rows, t.cols, block, stream);
        if (rc != BI8_OK) return rc;
    }
    return BI8_OK;
}

size_t bi8_peer_allreduce_buffer_bytes(int world, int64_t capacity) {
    if (world < 1 || world > 8 || capacity <= 0 || capacity % 1024 != 0) return 0;
    return peer_allreduce_buffer_bytes(world, capacity);
}

int bi8_peer_allreduce(void* const* peer_bufs, int rank, int world, int64_t capacity, const float* partial, int64_t M, int64_t N,
                       const void* bias, int bias_dtype, void* out, int out_dtype, unsigned wait_limit_us, void* stream) {
    if (!peer_bufs || !partial || !out) return fail(BI8_ERR_NULL, "peer all-reduce: null pointer");
    if (!dtype_ok(out_dtype) || (bias && !dtype_ok(bias_dtype & ~BI8_ADDEND_FULL))) return fail(BI8_ERR_DTYPE, "peer all-reduce: unknown dtype code");
    return launch_peer_allreduce(peer_bufs, rank, world, capacity, partial, M, N, bias, bias_dtype, out, out_dtype, wait_limit_us,
                                 static_cast<cudaStream_t>(stream));
}

int bi8_dequantize_rowwise_pitched(const int8_t* q, int64_t ldq, const float* s, void* out, int out_dtype, int64_t M, int64_t K, int block,
                                   void* stream) {
    DeviceOfCall call;
    if (!dtype_ok(out_dtype)) return fail(BI8_ERR_DTYPE, "dequantize: unknown dtype code %d", out_dtype);
    if (block < 1) return fail(BI8_ERR_BLOCK, "dequantize: block size %d", block);
    if (M < 0 || K < 0 || ldq < K) return fail(BI8_ERR_SHAPE, "dequantize: bad shape M=%lld K=%lld ldq=%lld", (long long)M, (long long)K, (long long)ldq);
    if (M == 0 || K == 0) return BI8_OK;
    if (!q || !s || !out) return fail(BI8_ERR_NULL, "dequantize: null pointer");
    if (!aligned(out, dtype_size(out_dtype)) || !aligned(s, 4)) return fail(BI8_ERR_ALIGN, "dequantize: pointer not element aligned");
    return launch_dequantize_rowwise(q, ldq, s, out, out_dtype, M, K, block, static_cast<cudaStream_t>(stream));
}

int bi8_dequantize_rowwise(const int8_t* q, const float* s, void* out, int out_dtype, int64_t M, int64_t K, int block,
                           void* stream) {
    return bi8_dequantize_rowwise_pitched(q, K, s, out, out_dtype, M, K, block, stream);
}

int bi8_copy_rows(const int8_t* src, int64_t lds, int8_t* dst, int64_t ldd, int64_t rows, int64_t cols, void* stream) {
    if (rows < 0 || cols < 0 || lds < cols || ldd < cols)
        return fail(BI8_ERR_SHAPE, "copy_rows: bad shape rows=%lld cols=%lld pitches %lld, %lld", (long long)rows, (long long)cols, (long long)lds, (long long)ldd);
    if (rows == 0 || cols == 0) return BI8_OK;
    if (!src || !dst) return fail(BI8_ERR_NULL, "copy_rows: null pointer");
    if (!aligned(dst, 16) || ldd % 16 != 0) return fail(BI8_ERR_ALIGN, "copy_rows: the copy's rows must begin on 16-byte boundaries");
    return launch_copy_rows(src, lds, dst, ldd, rows, cols, static_cast<cudaStream_t>(stream));
}

size_t bi8_column_sum_workspace_bytes(int64_t R, int64_t C) { return column_sum_workspace_bytes(R, C); }

int bi8_column_sum(const void* x, int dtype, int64_t ldx, void* out, int64_t R, int64_t C, void* workspace, size_t workspace_bytes, void* stream) {
    DeviceOfCall call;
    if (!dtype_ok(dtype)) return fail(BI8_ERR_DTYPE, "column_sum: unknown dtype code %d", dtype);
    if (R < 0 || C < 0 || ldx < C) return fail(BI8_ERR_SHAPE, "column_sum: bad shape R=%lld C=%lld ldx=%lld", (long long)R, (long long)C, (long long)ldx);
    if (C == 0) return BI8_OK;
    if (!out || (!x && R > 0)) return fail(BI8_ERR_NULL, "column_sum: null pointer");
    if (!aligned(x, dtype_size(dtype)) || !aligned(out, dtype_size(dtype))) return fail(BI8_ERR_ALIGN, "column_sum: pointer not element aligned");
    return launch_column_sum(x, dtype, ldx, out, R, C, workspace, workspace_bytes, static_cast<cudaStream_t>(stream));
}

namespace {
size_t gemm_scratch(int64_t M, int64_t N, int64_t K, int block, bool used) {
    DeviceOfCall call;
    if (M <= 0 || N <= 0 || K <= 0 || (block != 32 && block != 64 && block != 128)) return 0;
    GemmArgs g{};
    g.M = M;
    g.N = N;
    g.K = K;
    g.block = block;
    return gemm_tc_workspace_bytes(g, used);
}
}  // namespace

size_t bi8_gemm_workspace_bytes(int64_t M, int64_t N, int64_t K, int block) { return gemm_scratch(M, N, K, block, false); }
size_t bi8_gemm_workspace_used(int64_t M, int64_t N, int64_t K, int block) { return gemm_scratch(M, N, K, block, true); }

int bi8_gemm_dequant(const int8_t* A, int64_t lda, const int8_t* Bt, int64_t ldb, const float* sA, const float* sB,
                     const void* bias, int bias_dtype, void* C, int64_t ldc, int out_dtype, int64_t M, int64_t N, int64_t K,
                     int block, void* workspace, size_t workspace_bytes, int flags, void* stream) {
    DeviceOfCall call;
    GemmArgs g{A, lda, Bt, ldb, sA, sB, bias, bias_dtype, C, ldc, out_dtype, nullptr, M, N, K, block, flags, workspace, workspace_bytes};
    int rc = check_gemm(g, false);
    if (rc != BI8_OK || M == 0 || N == 0) return rc;
    return dispatch_gemm(g, static_cast<cudaStream_t>(stream));
}

int bi8_gemm_dequant_residual(const int8_t* A, int64_t lda, const int8_t* Bt, int64_t ldb, const float* sA, const float* sB, const void* bias,
                              int bias_dtype, const void* residual, int64_t ldr, void* C, int64_t ldc, int out_dtype, int64_t M, int64_t N,
                              int64_t K, int block, void* workspace, size_t workspace_bytes, int flags, void* stream) {
    DeviceOfCall call;
    GemmArgs g{A, lda, Bt, ldb, sA, sB, bias, bias_dtype, C, ldc, out_dtype, nullptr, M, N, K, block, flags, workspace, workspace_bytes};
    int rc = check_gemm(g, false);
    if (rc != BI8_OK || M == 0 || N == 0) return rc;
    if (residual && ldr < N) return fail(BI8_ERR_SHAPE, "gemm_dequant_residual: residual row pitch smaller than the row");
    if (residual && !aligned(residual, dtype_size(out_dtype))) return fail(BI8_ERR_ALIGN, "gemm_dequant_residual: residual not element aligned");
    if (overlaps_output(residual, ldr, C, ldc, out_dtype, M, N)) return fail(BI8_ERR_SHAPE, "gemm_dequant_residual: residual and C overlap");
    g.residual = residual;
    g.ldr = ldr;
    return dispatch_gemm(g, static_cast<cudaStream_t>(stream));
}

int bi8_gemm_block_partials(const int8_t* A, int64_t lda, const int8_t* Bt, int64_t ldb, int32_t* P, int64_t M, int64_t N,
                            int64_t K, int block, int flags, void* stream) {
    GemmArgs g{A, lda, Bt, ldb, nullptr, nullptr, nullptr, 0, nullptr, N, BI8_F32, P, M, N, K, block, flags, nullptr, 0};
    int rc = check_gemm(g, true);
    if (rc != BI8_OK || M == 0 || N == 0 || K == 0) return rc;
    return dispatch_gemm(g, static_cast<cudaStream_t>(stream));
}

int bi8_gemm_dequant_fused_quant(const void* x, int x_dtype, int64_t ldx, int8_t* xq, float* sx, const int8_t* Wq, int64_t ldw,
                                 const float* sW, const void* bias, int bias_dtype, void* C, int64_t ldc, int out_dtype,
                                 int64_t M, int64_t N, int64_t K, int block, void* workspace, size_t workspace_bytes, int flags,
                                 void* stream) {
    DeviceOfCall call;
    if (!dtype_ok(x_dtype)) return fail(BI8_ERR_DTYPE, "gemm_dequant_fused_quant: unknown dtype code %d", x_dtype);
    const bool forced = (flags & (BI8_GEMM_FORCE_GENERIC | BI8_GEMM_FORCE_TC | BI8_GEMM_FORCE_SMALLM)) != 0;
    if (!forced && x && M > 0 && N > 0 && K > 0 && ldx >= K && aligned(x, dtype_size(x_dtype)) && Wq && sW && C && ldw >= K && ldc >= N &&
        dtype_ok(out_dtype) && (!bias || dtype_ok(bias_dtype)) && aligned(C, dtype_size(out_dtype))) {
        const GemmArgs g{xq, K, Wq, ldw, sx, sW, bias, bias_dtype, C, ldc, out_dtype, nullptr, M, N, K, block, flags, workspace, workspace_bytes};
        bool done = false;
        const int rc = launch_decode(g, true, BI8_PRE_NONE, x, nullptr, nullptr, x_dtype, ldx, 0.0f, &done, static_cast<cudaStream_t>(stream));
        if (done) return rc;
    }
    // ... two kernels otherwise, through the caller's scratch
    if (M > 0 && K > 0 && (!xq || !sx))
        return fail(BI8_ERR_WORKSPACE, "gemm_dequant_fused_quant: this shape runs as quantize + GEMM and needs the xq / sx scratch");
    int rc = bi8_quantize_rowwise(x, x_dtype, ldx, xq, sx, M, K, block, stream);
    if (rc != BI8_OK) return rc;
    return bi8_gemm_dequant(xq, K, Wq, ldw, sx, sW, bias, bias_dtype, C, ldc, out_dtype, M, N, K, block, workspace,
                            workspace_bytes, flags & ~BI8_GEMM_FORCE_SKINNY, stream);
}

int bi8_quantize_rowwise_pre_pitched(int op, const void* x, const void* x2, int x_dtype, int64_t ldx, const void* weight, float eps, int8_t* q,
                                     int64_t ldq, float* scales, int64_t M, int64_t K, int block, void* stream) {
    DeviceOfCall call;
    if (!dtype_ok(x_dtype)) return fail(BI8_ERR_DTYPE, "quantize_rowwise_pre: unknown dtype code %d", x_dtype);
    if (op != BI8_PRE_NONE && op != BI8_PRE_RMSNORM && op != BI8_PRE_SILU_MUL)
        return fail(BI8_ERR_SHAPE, "quantize_rowwise_pre: unknown operation code %d", op);
    if (M < 0 || K < 0 || ldx < K || ldq < K) return fail(BI8_ERR_SHAPE, "quantize_rowwise_pre: bad shape M %lld K %lld ldx %lld", (long long)M, (long long)K, (long long)ldx);
    if (M == 0 || K == 0) return BI8_OK;
    if (!x || !q || !scales || (op == BI8_PRE_SILU_MUL && !x2)) return fail(BI8_ERR_NULL, "quantize_rowwise_pre: null pointer");
    const size_t esz = dtype_size(x_dtype);
    if (!aligned(x, esz) || (x2 && !aligned(x2, esz)) || (weight && !aligned(weight, esz)) || !aligned(scales, 4))
        return fail(BI8_ERR_ALIGN, "quantize_rowwise_pre: pointer not element aligned");
    return launch_quantize_pre(op, x, x2, x_dtype, ldx, weight, eps, q, ldq, scales, M, K, block, static_cast<cudaStream_t>(stream));
}

int bi8_quantize_rowwise_pre(int op, const void* x, const void* x2, int x_dtype, int64_t ldx, const void* weight, float eps, int8_t* q,
                             float* scales, int64_t M, int64_t K, int block, void* stream) {
    return bi8_quantize_rowwise_pre_pitched(op, x, x2, x_dtype, ldx, weight, eps, q, K, scales, M, K, block, stream);
}

int bi8_gemm_dequant_fused_pre(int op, const void* x, const void* x2, int x_dtype, int64_t ldx, const void* norm_weight, float eps,
                               int8_t* xq, float* sx, const int8_t* Wq, int64_t ldw, const float* sW, const void* bias, int bias_dtype,
                               const void* residual, int64_t ldr, void* C, int64_t ldc, int out_dtype, int64_t M, int64_t N, int64_t K,
                               int block, void* workspace, size_t workspace_bytes, int flags, void* stream) {
    DeviceOfCall call;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool scratch = xq != nullptr && sx != nullptr;
    if (residual && ldr < N) return fail(BI8_ERR_SHAPE, "gemm_dequant_fused_pre: residual row pitch smaller than the row");
    if (!dtype_ok(out_dtype)) return fail(BI8_ERR_DTYPE, "gemm_dequant_fused_pre: unknown output dtype code %d", out_dtype);
    if (residual && !aligned(residual, dtype_size(out_dtype))) return fail(BI8_ERR_ALIGN, "gemm_dequant_fused_pre: residual not element aligned");
    if (M == 0 || N == 0) return BI8_OK;
    const bool overlap = overlaps_output(residual, ldr, C, ldc, out_dtype, M, N);
    if (overlap && (residual != C || ldr != ldc))
        return fail(BI8_ERR_SHAPE, "gemm_dequant_fused_pre: residual and C overlap without being the same tensor");
    if (op == BI8_PRE_NONE && !residual)
        return bi8_gemm_dequant_fused_quant(x, x_dtype, ldx, xq, sx, Wq, ldw, sW, bias, bias_dtype, C, ldc, out_dtype, M, N, K, block,
                                            workspace, workspace_bytes, flags, stream);
    // the decode path: this op's quantizer in the decode quantizer's place, the GEMM overlapped with it, the residual
    // added by the kernel that writes C (through the bias operand, which gets a row pitch)
    const bool forced = (flags & (BI8_GEMM_FORCE_GENERIC | BI8_GEMM_FORCE_TC | BI8_GEMM_FORCE_SMALLM)) != 0;
    GemmArgs g{xq, K, Wq, ldw, sx, sW, bias, bias_dtype, C, ldc, out_dtype, nullptr, M, N, K, block, flags, workspace, workspace_bytes};
    const bool x_ok = x && dtype_ok(x_dtype) && ldx >= K && aligned(x, dtype_size(x_dtype)) && (op != BI8_PRE_SILU_MUL || (x2 && aligned(x2, dtype_size(x_dtype)))) &&
                      (!norm_weight || aligned(norm_weight, dtype_size(x_dtype))) && (op == BI8_PRE_NONE || op == BI8_PRE_RMSNORM || op == BI8_PRE_SILU_MUL);
    const bool in_kernel_residual = residual && !bias;
    if (!forced && K > 0 && x_ok && !(overlap && !in_kernel_residual)) {
        int rc = check_gemm(g, false, scratch);
        if (rc != BI8_OK) return rc;
        if (in_kernel_residual) {
            g.bias = residual;
            g.bias_dtype = out_dtype;
            g.bias_ld = ldr;
        }
        bool done = false;
        rc = launch_decode(g, false, op, x, x2, norm_weight, x_dtype, ldx, eps, &done, st);
        if (done) {
            if (rc != BI8_OK || !residual || in_kernel_residual) return rc;
            return launch_residual_add(C, ldc, residual, ldr, out_dtype, M, N, st);
        }
        g.bias_ld = 0;
    }
    if (K > 0 && !scratch)
        return fail(BI8_ERR_WORKSPACE, "gemm_dequant_fused_pre: this shape runs as quantize + GEMM and needs the xq / sx scratch");
    // The general tensor-core kernel reads an element of the residual in the warp that then writes it, so C may be the residual.
    const char* why = "";
    if (overlap && ((flags & BI8_GEMM_FORCE_GENERIC) || bias || K == 0 || !gemm_tc_applicable(g, &why)))
        return fail(BI8_ERR_ALIGN, "gemm_dequant_fused_pre: C may be the residual itself only for the tensor-core kernels, without bias");
    if (overlap) flags |= BI8_GEMM_FORCE_TC;
    int rc = bi8_quantize_rowwise_pre(op, x, x2, x_dtype, ldx, norm_weight, eps, xq, sx, M, K, block, stream);
    if (rc != BI8_OK) return rc;
    g.flags = flags & ~BI8_GEMM_QUANT_IN_KERNEL;
    g.bias = bias;
    g.bias_dtype = bias_dtype;
    g.residual = residual;
    g.ldr = ldr;
    rc = check_gemm(g, false);
    return rc != BI8_OK ? rc : dispatch_gemm(g, st);
}

size_t bi8_peer_allreduce_large_buffer_bytes(int world, int64_t capacity) {
    if (world < 1 || world > 8 || capacity <= 0 || capacity % 1024 != 0) return 0;
    return peer_allreduce_large_buffer_bytes(capacity);
}

size_t bi8_peer_allreduce_large_partial_offset(void) { return peer_allreduce_large_partial_offset(); }

size_t bi8_peer_allreduce_large_out_offset(int64_t capacity) { return peer_allreduce_large_out_offset(capacity); }

int bi8_peer_allreduce_large(void* const* peer_bufs, int rank, int world, int64_t capacity, int64_t M, int64_t N, const void* bias,
                             int bias_dtype, int out_dtype, unsigned wait_limit_us, void* stream) {
    if (!peer_bufs) return fail(BI8_ERR_NULL, "peer all-reduce: null pointer");
    if (!dtype_ok(out_dtype) || (bias && !dtype_ok(bias_dtype & ~BI8_ADDEND_FULL))) return fail(BI8_ERR_DTYPE, "peer all-reduce: unknown dtype code");
    return launch_peer_allreduce_large(peer_bufs, rank, world, capacity, M, N, bias, bias_dtype, out_dtype, wait_limit_us,
                                       static_cast<cudaStream_t>(stream));
}

int bi8_row_parallel_linear_pre(int op, const void* x, const void* x2, int x_dtype, int64_t ldx, const void* norm_weight, float eps,
                                int8_t* xq, float* sx, const int8_t* Wq, int64_t ldw, const float* sW, float* partial, int64_t M, int64_t N,
                                int64_t K, int block, void* workspace, size_t workspace_bytes, void* const* peer_bufs, int rank, int world,
                                int64_t capacity, const void* bias, int bias_dtype, void* out, int out_dtype, unsigned wait_limit_us,
                                int flags, void* stream) {
    if (!x || !xq || !sx || !Wq || !sW || !partial || !peer_bufs || !out) return fail(BI8_ERR_NULL, "row_parallel_linear: null pointer");
    if (!dtype_ok(x_dtype) || !dtype_ok(out_dtype) || (bias && !dtype_ok(bias_dtype & ~BI8_ADDEND_FULL)))
        return fail(BI8_ERR_DTYPE, "row_parallel_linear: unknown dtype code");
    if (M <= 0 || N <= 0 || K <= 0 || ldx < K || ldw < K) return fail(BI8_ERR_SHAPE, "row_parallel_linear: bad shape M=%lld N=%lld K=%lld", (long long)M, (long long)N, (long long)K);
    if (!aligned(partial, 16) || !aligned(out, 16)) return fail(BI8_ERR_ALIGN, "row_parallel_linear: partial and out must be 16-byte aligned");
    PeerArgs pa;
    int rc = make_peer_args(&pa, peer_bufs, rank, world, capacity, M, N);
    if (rc != BI8_OK) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool forced = (flags & (BI8_GEMM_FORCE_GENERIC | BI8_GEMM_FORCE_TC | BI8_GEMM_FORCE_SMALLM | BI8_GEMM_QUANT_IN_KERNEL)) != 0;
    const bool x_vec = aligned(x, 16) && (ldx * dtype_size(x_dtype)) % 16 == 0;
    if (!forced && (x_vec || op != BI8_PRE_NONE) && K % 16 == 0 && aligned(xq, 16)) {
        // decode-sized M: quantizer, weight-streaming GEMM into `partial`, and a kernel behind it that sums the ranks
        GemmArgs g{xq, K, Wq, ldw, sx, sW, nullptr, 0, partial, N, BI8_F32, nullptr, M, N, K, block, flags, workspace, workspace_bytes};
        if (gemm_skinny_applicable(g)) {
            PeerEpilogue pe{&pa, bias, bias_dtype, out, out_dtype, peer_wait_limit_cycles(wait_limit_us)};
            if (op == BI8_PRE_NONE) rc = launch_skinny_quantize(x, x_dtype, ldx, xq, sx, M, K, block, st);
            else rc = bi8_quantize_rowwise_pre(op, x, x2, x_dtype, ldx, norm_weight, eps, xq, sx, M, K, block, stream);
            if (rc != BI8_OK) return rc;
            g.after_own_quantizer = true;
            g.peer = &pe;
            return launch_gemm_skinny(g, st);
        }
    }
    // other shapes: the layer's two steps into `partial`, then the stand-alone reduction
    rc = bi8_gemm_dequant_fused_pre(op, x, x2, x_dtype, ldx, norm_weight, eps, xq, sx, Wq, ldw, sW, nullptr, 0, nullptr, 0, partial, N,
                                    BI8_F32, M, N, K, block, workspace, workspace_bytes, flags, stream);
    if (rc != BI8_OK) return rc;
    return launch_peer_allreduce(peer_bufs, rank, world, capacity, partial, M, N, bias, bias_dtype, out, out_dtype, wait_limit_us, st);
}

int bi8_row_parallel_linear(const void* x, int x_dtype, int64_t ldx, int8_t* xq, float* sx, const int8_t* Wq, int64_t ldw,
                            const float* sW, float* partial, int64_t M, int64_t N, int64_t K, int block, void* workspace,
                            size_t workspace_bytes, void* const* peer_bufs, int rank, int world, int64_t capacity, const void* bias,
                            int bias_dtype, void* out, int out_dtype, unsigned wait_limit_us, int flags, void* stream) {
    return bi8_row_parallel_linear_pre(BI8_PRE_NONE, x, nullptr, x_dtype, ldx, nullptr, 0.0f, xq, sx, Wq, ldw, sW, partial, M, N, K, block,
                                       workspace, workspace_bytes, peer_bufs, rank, world, capacity, bias, bias_dtype, out, out_dtype,
                                       wait_limit_us, flags, stream);
}

int bi8_rope_cache_append(const void* qkv, int dtype, const float* cis, const long long* pos, void* q_out, void* kcache, void* vcache,
                          int64_t B, int64_t H, int64_t D, int64_t max_len, void* stream) {
    if (dtype != BI8_BF16 && dtype != BI8_F16) return fail(BI8_ERR_DTYPE, "rope_cache_append: bf16 or fp16 activations (got code %d)", dtype);
    if (B < 0 || H < 0 || D < 0 || D % 2 != 0 || max_len <= 0 || B > 0x7fffffff || H > 0x7fffffff || D > 0x7fffffff || max_len > 0x7fffffff)
        return fail(BI8_ERR_SHAPE, "rope_cache_append: bad shape B %lld H %lld D %lld max_len %lld", (long long)B, (long long)H, (long long)D, (long long)max_len);
    if (B == 0 || H == 0 || D == 0) return BI8_OK;
    if (!qkv || !cis || !pos || !q_out || !kcache || !vcache) return fail(BI8_ERR_NULL, "rope_cache_append: null pointer");
    if (!aligned(qkv, 4) || !aligned(q_out, 4) || !aligned(kcache, 4) || !aligned(vcache, 4) || !aligned(cis, 8) || !aligned(pos, 8))
        return fail(BI8_ERR_ALIGN, "rope_cache_append: pointer not aligned to an element pair");
    return launch_rope_cache_append(qkv, dtype, cis, pos, q_out, kcache, vcache, B, H, D, max_len, static_cast<cudaStream_t>(stream));
}

int bi8_stream_capture_id(void* stream, unsigned long long* id) {
    if (!id) return fail(BI8_ERR_NULL, "stream_capture_id: null output");
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    unsigned long long cid = 0;
    BI8_CUDA_TRY(cudaStreamGetCaptureInfo(static_cast<cudaStream_t>(stream), &st, &cid));
    *id = (st == cudaStreamCaptureStatusActive) ? cid : 0ull;
    return BI8_OK;
}

int bi8_gemm_wait_selftest(const int8_t* A, int64_t lda, const int8_t* Bt, int64_t ldb, const float* sA, const float* sB, void* C,
                           int64_t ldc, int out_dtype, int64_t M, int64_t N, int64_t K, int block, unsigned wait_limit_us,
                           int skip_stage, void* stream) {
    GemmArgs g{A, lda, Bt, ldb, sA, sB, nullptr, 0, C, ldc, out_dtype, nullptr, M, N, K, block, BI8_GEMM_FORCE_TC, nullptr, 0};
    int rc = check_gemm(g, false);
    if (rc != BI8_OK) return rc;
    if (M == 0 || N == 0 || K == 0) return fail(BI8_ERR_SHAPE, "gemm_wait_selftest: empty problem");
    if (wait_limit_us > 2000000u) return fail(BI8_ERR_LIMIT, "gemm_wait_selftest: wait limit above two seconds");
    g.wait_limit_us = wait_limit_us;
    g.skip_stage = skip_stage;
    return dispatch_gemm(g, static_cast<cudaStream_t>(stream));
}

int bi8_mma_peak_probe(int iters, float* ms, int* sm_count) {
    if (!ms) return fail(BI8_ERR_NULL, "mma_peak_probe: null output");
    return run_mma_peak_probe(iters, ms, sm_count);
}

}  // extern "C"
