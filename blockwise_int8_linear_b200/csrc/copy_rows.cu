// Copy of int8 rows of any alignment to rows that begin on 16-byte boundaries.
//
// The tensor-core GEMM reads its operands by TMA, which takes rows on 16-byte boundaries only.  The library's own intermediate results
// have them; a dense int8 matrix whose rows are not a multiple of 16 long (the weight buffer of such a layer, a checkpoint's
// copy, a caller's own tensor) is copied once per call.  Bound by memory, and for the matrices of a few hundred KB that occur by the
// latency of a launch: 777 x 1000 takes 2 us, 9 us with the three tensor operations that it replaces.  (copy_rows.cuh has
// what a thread does; beside a layer's activations it shares their quantizer's launch: quantize_jobs_kernel in quantize.cu.)
#include "bi8_common.cuh"
#include "copy_rows.cuh"

namespace bi8 {
namespace {

constexpr int kCopyThreads = 256;

__global__ void __launch_bounds__(kCopyThreads) copy_rows_kernel(const int8_t* __restrict__ src, int64_t lds, int8_t* __restrict__ dst, int64_t ldd,
                                                                 int64_t pieces, int per_row, int64_t cols) {
    after_predecessor();
    const int64_t i = (int64_t)blockIdx.x * kCopyThreads + threadIdx.x;
    copy_rows_piece(i, src, lds, dst, ldd, pieces, per_row, cols);
}

}  // namespace

int launch_copy_rows(const int8_t* src, int64_t lds, int8_t* dst, int64_t ldd, int64_t rows, int64_t cols, cudaStream_t st) {
    const int64_t per_row = (cols + 15) / 16;
    if (per_row > 0x7fffffff) return fail(BI8_ERR_LIMIT, "copy_rows: rows longer than 2^35");
    const int64_t pieces = rows * per_row, grid = (pieces + kCopyThreads - 1) / kCopyThreads;
    if (grid > 0x7fffffff) return fail(BI8_ERR_LIMIT, "copy_rows: more than 2^31 blocks");
    return launch_chained(copy_rows_kernel, (unsigned)grid, kCopyThreads, 0, st, src, lds, dst, ldd, pieces, (int)per_row, cols);
}

}  // namespace bi8
