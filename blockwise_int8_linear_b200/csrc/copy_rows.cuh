// What a thread of a copy of int8 rows to 16-byte boundaries does: 16 bytes of a row from the two aligned pieces that hold them; its
// neighbour reads the second one too, from L1.
#pragma once

#include "bi8_common.cuh"

#include <type_traits>

namespace bi8 {

__device__ __forceinline__ void copy_rows_piece(int64_t i, const int8_t* __restrict__ src, int64_t lds, int8_t* __restrict__ dst, int64_t ldd,
                                                int64_t pieces, int per_row, int64_t cols) {
    if (i >= pieces) return;
    const int64_t row = i / per_row, c = (i - row * per_row) * 16;
    const uintptr_t a = reinterpret_cast<uintptr_t>(src + row * lds + c), end = reinterpret_cast<uintptr_t>(src + row * lds + cols);
    const uintptr_t base = a & ~(uintptr_t)15;
    // a piece is read only where it holds a byte of the row: no access leaves the matrix's 16-byte granules
    const uint4 lo = __ldg(reinterpret_cast<const uint4*>(base));
    uint4 hi = make_uint4(0u, 0u, 0u, 0u);
    if (base + 16 < end) hi = __ldg(reinterpret_cast<const uint4*>(base + 16));
    const uint32_t r[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    const uint32_t off = (uint32_t)(a & 15u), bits = (off & 3u) * 8u;
    uint32_t w[4];
    auto shifted = [&](auto words) {
        constexpr int WS = decltype(words)::value;
#pragma unroll
        for (int k = 0; k < 4; ++k) w[k] = __funnelshift_r(r[k + WS], r[k + WS + 1], bits);
    };
    if (off < 4u) shifted(std::integral_constant<int, 0>{});
    else if (off < 8u) shifted(std::integral_constant<int, 1>{});
    else if (off < 12u) shifted(std::integral_constant<int, 2>{});
    else shifted(std::integral_constant<int, 3>{});
    *reinterpret_cast<uint4*>(dst + row * ldd + c) = make_uint4(w[0], w[1], w[2], w[3]);
}

}  // namespace bi8
