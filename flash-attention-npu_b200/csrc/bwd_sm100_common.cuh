// Pieces shared by the tcgen05 backward kernels (head dims up to 128: bwd_sm100.cu; above: bwd_wide_sm100.cu).
#pragma once
#include "fa_utils.cuh"
#include "fa_internal.h"
#include "sm100_ptx.cuh"

namespace fa {

// 32 accumulator columns -> the row, scaled and rounded; `left` = columns of the row that remain from dst on (the
// kernels run a padded head dim, the row holds the call's own)
template <typename T>
__device__ __forceinline__ void store_row_scaled(T* dst, const uint32_t (&r)[32], float s, int left) {
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        if (v * 8 >= left) break;
        uint4 pk;
        pk.x = Elem<T>::pack(__uint_as_float(r[8 * v + 0]) * s, __uint_as_float(r[8 * v + 1]) * s);
        pk.y = Elem<T>::pack(__uint_as_float(r[8 * v + 2]) * s, __uint_as_float(r[8 * v + 3]) * s);
        pk.z = Elem<T>::pack(__uint_as_float(r[8 * v + 4]) * s, __uint_as_float(r[8 * v + 5]) * s);
        pk.w = Elem<T>::pack(__uint_as_float(r[8 * v + 6]) * s, __uint_as_float(r[8 * v + 7]) * s);
        reinterpret_cast<uint4*>(dst)[v] = pk;
    }
}

}  // namespace fa
