// Bit-packed node types: the set-up kernels (boundary points, lattice
// construction) read the fluid points as one bit each, 32 along an axis to a
// word.  A 512x1024x512 grid is 34 MB instead of 268 MB of bytes, and runs,
// dilations and ranks become word operations.
//
// Set-up of the vascular tree on that grid, byte arrays against bits: boundary
// points 840 -> 47 us; lattice (axis choice, types, ids, pieces, masks) 24 -> 1.7
// ms of kernels; the whole set-up call 56 -> 25 ms.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace lbm {

__host__ __device__ constexpr int words_for(int n) { return (n + 31) >> 5; }

// Value of grid point p (x-major, columns of Nz points) in bits of W words a column.
__host__ __device__ __forceinline__ uint8_t point_bit(const uint32_t* bits, int64_t p, int W, int Nz) {
    const int64_t col = p / Nz;
    const int k = (int)(p - col * Nz);
    return (uint8_t)((bits[col * W + (k >> 5)] >> (k & 31)) & 1u);
}

// 32x32 bits per warp: lane l gives row l, receives column l
__device__ __forceinline__ uint32_t transpose32(uint32_t v) {
    const int lane = threadIdx.x & 31;
    uint32_t out = 0;
#pragma unroll
    for (int b = 0; b < 32; ++b) {
        const uint32_t w = __ballot_sync(0xffffffffu, (v >> b) & 1u);
        if (lane == b) out = w;
    }
    return out;
}

// Calls fn(word index, word, bit, set, rank) for every nonzero word of [0, n), all
// lanes of the warp together, lane l for bit l; rank: prefix[word] + set bits
// below.  A warp takes 32 words.
template <class F>
__device__ __forceinline__ void for_each_bit(const uint32_t* __restrict__ words, const uint32_t* __restrict__ prefix, int64_t n,
                                             F fn) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t b = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * 32; b < n; b += nw * 32) {
        const uint32_t mine = b + lane < n ? words[b + lane] : 0u;
        const uint32_t pre = b + lane < n && mine ? prefix[b + lane] : 0u;
        for (unsigned m = __ballot_sync(0xffffffffu, mine != 0u); m; m &= m - 1) {
            const int src = __ffs(m) - 1;
            const uint32_t w = __shfl_sync(0xffffffffu, mine, src);
            const uint32_t p = __shfl_sync(0xffffffffu, pre, src);
            fn(b + src, w, lane, (w >> lane) & 1u, p + __popc(w & ((1u << lane) - 1u)));
        }
    }
}

}  // namespace lbm
