// Grid columns between two FP32 cell coordinates (voxelizer).
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define LBM_HD __host__ __device__ __forceinline__
#else
#define LBM_HD inline
#endif

namespace lbm {

// Last of n columns at or below hi (any number but NaN, above -2^31), negative if
// there is none.  Compared as integers: n - 1 is not a float beyond 2^24.
LBM_HD int last_column(float hi, int n) {
    const int i = hi < 2147483648.f ? (int)floorf(hi) : n - 1;
    return i < n - 1 ? i : n - 1;
}

}  // namespace lbm
