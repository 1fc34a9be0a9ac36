// mode_index.cuh -- the (j, k) of a mode of one i plane, for the per-mode update (host and device).
#pragma once

namespace pd {

#if defined(__CUDACC__)
#define PD_MODE_HD __host__ __device__ __forceinline__
#else
#define PD_MODE_HD inline
#endif

// Longest transform length, and the modes of the largest plane (NKJ NKK) it allows.
constexpr int kMaxLength = 1024;
constexpr int kMaxPlane = (2 * (kMaxLength / 3) + 1) * (2 * (kMaxLength / 3) + 1);
static_assert(kMaxPlane < (1 << 19), "mode_row is exact below 2^19 modes");

// Mode q = j NKK + k of a plane: j from a product with 1 / NKK in 32-bit floating point, exact
// for planes below 2^19 modes (0.5 / NKK is more than twice its rounding).
PD_MODE_HD void mode_row(int q, int nkk, int& j, int& k) {
    j = (int)(((float)q + 0.5f) * (1.0f / (float)nkk));
    k = q - j * nkk;
}

}  // namespace pd
