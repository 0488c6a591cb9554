// Sum over the rows of a matrix, out[c] = cast(sum_r x[r, c]) in fp32: the bias gradient of a layer (block_linear.py:105-106 in
// the reference, where torch sums).
//
// Bound by reading x once (from L2 where the gradient's quantizer has just read it).  A CTA takes 128 columns (16 threads x 8
// columns, one 16-byte load of a 16-bit row each; two for fp32) of a range of rows, 16 rows at a time, eight steps of loads in
// flight; the row lanes meet in shared memory in a fixed order.  There are as many row ranges as fill the device;
// their fp32 sums go to a workspace and a second kernel adds them in ascending order, so the result does not depend on
// scheduling.  (torch's reduction over the leading dimension: 29 us for 8192 x 3072 bf16, 8 us of host time per call.)
#include "bi8_common.cuh"
#include "tc_common.cuh"

namespace bi8 {
namespace {

constexpr int kSumCols = 128, kSumThreads = 256, kSumLanes = kSumThreads / (kSumCols / 8);

template <int DT>
__device__ __forceinline__ float sum_load1(const void* x, int64_t i) {
    if (DT == BI8_F32) return static_cast<const float*>(x)[i];
    const unsigned short h = static_cast<const unsigned short*>(x)[i];
    return DT == BI8_BF16 ? bf16lo(h) : __half2float(__ushort_as_half(h));
}

// eight columns of a row; `live` of them exist
template <int DT>
__device__ __forceinline__ void sum_load8(float (&f)[8], const void* x, int64_t i, int live, bool vec) {
    if (vec && live >= 8) {
        if (DT == BI8_F32) {
            const uint4 a = ld_nc_v4(static_cast<const float*>(x) + i), b = ld_nc_v4(static_cast<const float*>(x) + i + 4);
            f[0] = __uint_as_float(a.x); f[1] = __uint_as_float(a.y); f[2] = __uint_as_float(a.z); f[3] = __uint_as_float(a.w);
            f[4] = __uint_as_float(b.x); f[5] = __uint_as_float(b.y); f[6] = __uint_as_float(b.z); f[7] = __uint_as_float(b.w);
        } else {
            const uint4 a = ld_nc_v4(static_cast<const unsigned short*>(x) + i);
            const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                if (DT == BI8_BF16) {
                    f[2 * h] = bf16lo(w[h]);
                    f[2 * h + 1] = bf16hi(w[h]);
                } else {
                    const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&w[h]));
                    f[2 * h] = t.x;
                    f[2 * h + 1] = t.y;
                }
            }
        }
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = e < live ? sum_load1<DT>(x, i + e) : 0.0f;
    }
}

__device__ __forceinline__ void sum_store(void* out, int dt, int64_t c, float v) {
    if (dt == BI8_BF16) static_cast<__nv_bfloat16*>(out)[c] = __float2bfloat16_rn(v);
    else if (dt == BI8_F16) static_cast<__half*>(out)[c] = __float2half_rn(v);
    else static_cast<float*>(out)[c] = v;
}

// partial == nullptr: one row range, the result is written directly
template <int DT>
__global__ void __launch_bounds__(kSumThreads) column_sum_kernel(const void* __restrict__ x, int64_t ldx, void* __restrict__ out,
                                                                 float* __restrict__ partial, int R, int C, int rows_per_range, int vec) {
    after_predecessor();
    __shared__ float s_sum[kSumLanes][kSumCols + 4];
    const int cv = threadIdx.x % (kSumCols / 8), lane = threadIdx.x / (kSumCols / 8);
    const int c0 = blockIdx.x * kSumCols + cv * 8, live = C - c0;
    const int r0 = blockIdx.y * rows_per_range, r1 = r0 + rows_per_range < R ? r0 + rows_per_range : R;
    float acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.0f;
    if (live > 0) {
        constexpr int STEPS = 8;
        int r = r0 + lane;
        if (vec && live >= 8) {
            for (; r + (STEPS - 1) * kSumLanes < r1; r += kSumLanes * STEPS) {      // no test between the loads
                float f[STEPS][8];
#pragma unroll
                for (int u = 0; u < STEPS; ++u) sum_load8<DT>(f[u], x, (int64_t)(r + u * kSumLanes) * ldx + c0, 8, true);
#pragma unroll
                for (int u = 0; u < STEPS; ++u)
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[e] += f[u][e];
            }
        }
        for (; r < r1; r += kSumLanes) {
            float f[8];
            sum_load8<DT>(f, x, (int64_t)r * ldx + c0, live, vec != 0);
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] += f[e];
        }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) s_sum[lane][cv * 8 + e] = acc[e];
    __syncthreads();
    const int c = blockIdx.x * kSumCols + threadIdx.x;
    if (threadIdx.x < kSumCols && c < C) {
        float v = 0.0f;
#pragma unroll
        for (int l = 0; l < kSumLanes; ++l) v += s_sum[l][threadIdx.x];
        if (partial) partial[(int64_t)blockIdx.y * C + c] = v;
        else sum_store(out, DT, c, v);
    }
}

__global__ void __launch_bounds__(128) column_sum_finish_kernel(const float* __restrict__ partial, void* __restrict__ out, int dt, int C, int ranges) {
    after_predecessor();
    const int c = blockIdx.x * 128 + threadIdx.x;
    if (c >= C) return;
    float v = 0.0f;
    for (int g0 = 0; g0 < ranges; g0 += 8) {
        float f[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) f[u] = g0 + u < ranges ? __ldcg(partial + (int64_t)(g0 + u) * C + c) : 0.0f;
#pragma unroll
        for (int u = 0; u < 8; ++u) v += f[u];
    }
    sum_store(out, dt, c, v);
}

// The same for many partial rows (one per 128 rows of the matrix): 32 columns by eight groups of consecutive partial rows, each in
// ascending order with eight loads in flight, then the groups in ascending order.
__global__ void __launch_bounds__(256) column_sum_groups_kernel(const float* __restrict__ partial, void* __restrict__ out, int dt, int C, int ranges) {
    after_predecessor();
    __shared__ float s_part[8][32];
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
    const int per = (ranges + 7) / 8, r0 = g * per, r1 = r0 + per < ranges ? r0 + per : ranges;
    float v = 0.0f;
    if (c < C) {
        for (int r = r0; r < r1; r += 8) {
            float f[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) f[u] = r + u < r1 ? __ldcg(partial + (int64_t)(r + u) * C + c) : 0.0f;
#pragma unroll
            for (int u = 0; u < 8; ++u) v += f[u];
        }
    }
    s_part[g][lane] = v;
    __syncthreads();
    if (g == 0 && c < C) {
        v = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) v += s_part[k][lane];
        sum_store(out, dt, c, v);
    }
}

// Row ranges: enough CTAs for four per SM, but at least 128 rows each, one batch of loads.
int row_ranges(int64_t R, int64_t C, int sms) {
    const int64_t ctiles = (C + kSumCols - 1) / kSumCols;
    int64_t n = (4ll * sms + ctiles - 1) / ctiles;
    if (n > (R + 127) / 128) n = (R + 127) / 128;
    if (n > 128) n = 128;
    return n < 1 ? 1 : (int)n;
}

}  // namespace

size_t column_sum_workspace_bytes(int64_t R, int64_t C) {
    const DeviceInfo di = device_info();
    if (di.sms <= 0 || R <= 0 || C <= 0) return 0;
    const int n = row_ranges(R, C, di.sms);
    return n > 1 ? (size_t)n * (size_t)C * 4 : 0;
}

int launch_column_sum(const void* x, int dt, int64_t ldx, void* out, int64_t R, int64_t C, void* workspace, size_t workspace_bytes, cudaStream_t st) {
    if (R >= (1ll << 31) - 65536 || C >= (1ll << 31) - 65536) return fail(BI8_ERR_LIMIT, "column_sum: R or C too large");
    const DeviceInfo di = device_info();
    int ranges = row_ranges(R, C, di.sms > 0 ? di.sms : 1);
    if (workspace == nullptr || workspace_bytes < (size_t)ranges * (size_t)C * 4 || !aligned(workspace, 4)) ranges = 1;
    const int rows = R > 0 ? (int)((R + ranges - 1) / ranges) : 1;
    ranges = R > 0 ? (int)((R + rows - 1) / rows) : 1;
    const unsigned ctiles = (unsigned)((C + kSumCols - 1) / kSumCols);
    const int vec = aligned(x, 16) && (ldx * (dt == BI8_F32 ? 4 : 2)) % 16 == 0;
    float* partial = ranges > 1 ? static_cast<float*>(workspace) : nullptr;
    auto launch = [&](auto kernel) {
        return launch_chained_grid(kernel, dim3(ctiles, (unsigned)ranges), kSumThreads, 0, st, x, ldx, out, partial, (int)R, (int)C, rows, vec);
    };
    const int rc = dt == BI8_BF16 ? launch(column_sum_kernel<BI8_BF16>) : dt == BI8_F16 ? launch(column_sum_kernel<BI8_F16>) : launch(column_sum_kernel<BI8_F32>);
    if (rc != BI8_OK || ranges == 1) return rc;
    return launch_chained(column_sum_finish_kernel, (unsigned)((C + 127) / 128), 128, 0, st, partial, out, dt, (int)C, ranges);
}

// Column sums of `ranges` partial rows [ranges, C].
int launch_column_sum_finish(const float* partial, void* out, int dt, int64_t C, int64_t ranges, cudaStream_t st) {
    if (C >= (1ll << 31) - 65536 || ranges >= (1ll << 31)) return fail(BI8_ERR_LIMIT, "column_sum: too many columns or partial sums");
    return launch_chained(column_sum_groups_kernel, (unsigned)((C + 31) / 32), 256, 0, st, partial, out, dt, (int)C, (int)ranges);
}

}  // namespace bi8
