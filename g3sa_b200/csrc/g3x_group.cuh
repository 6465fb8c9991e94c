// g3x_group.cuh -- steps of the group-per-job kernels (g3x_group16.cu, g3x_global.cu): a group of G
// lanes (a power of two, aligned) holds a row of int16x2 blocks, eight columns a lane.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "g3x_core.h"

namespace g3x {

constexpr unsigned kAll = 0xFFFFFFFFu;

// A decay of `steps` lanes for values held in the high half of a word; values stay below 2^15,
// so a decay of 2^15 - 1 already leaves nothing.
__device__ __forceinline__ int32_t decay_hi(int32_t e_ins, int steps) {
    const int32_t v = 8 * steps * e_ins;
    return -((v < 0x7FFF ? v : 0x7FFF) << 16);
}

// Largest of the group's values, in every lane of it.
template <int G>
__device__ __forceinline__ int32_t max_of_group(int32_t v) {
    if constexpr (G == 32) {
        return __reduce_max_sync(kAll, v);
    } else {
#pragma unroll
        for (int o = G / 2; o >= 1; o >>= 1) v = max(v, __shfl_xor_sync(kAll, v, o));
        return v;
    }
}

// Exclusive prefix over the lanes of a group of the F leaving each block (high halves of x): F
// entering the lane's block, where a value loses 8 e_ins per lane it passes.  A lane that a
// shuffle leaves alone meets its own value, less the decay.  For G = 32, where a row's latency
// counts, three lanes per step (four dependent shuffles instead of six).
template <int G>
__device__ __forceinline__ int32_t f_entering(int32_t x, int r, int32_t e_ins) {
    const int32_t y = __shfl_up_sync(kAll, x, 1, G);
    int32_t f = r ? y : 0;
    if constexpr (G < 32) {
#pragma unroll
        for (int o = 1; o < G; o <<= 1) f = __viaddmax_s32(__shfl_up_sync(kAll, f, o, G), decay_hi(e_ins, o), f);
    } else {
#pragma unroll
        for (int o = 1; o < 16; o <<= 2) {
            const int32_t a = __shfl_up_sync(kAll, f, o), b = __shfl_up_sync(kAll, f, 2 * o);
            const int32_t c = __shfl_up_sync(kAll, f, 3 * o);
            f = __viaddmax_s32(a, decay_hi(e_ins, o), f);
            f = __viaddmax_s32(b, decay_hi(e_ins, 2 * o), f);
            f = __viaddmax_s32(c, decay_hi(e_ins, 3 * o), f);
        }
        f = __viaddmax_s32(__shfl_up_sync(kAll, f, 16), decay_hi(e_ins, 16), f);
    }
    return f;
}

}  // namespace g3x
