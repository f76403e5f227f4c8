// Arithmetic of the prompt-column kernels that the CPU can hold to its definition: plain C++, device code under nvcc.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define MLB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define MLB_HOST_DEVICE inline
#endif

namespace mlb {

// x / sqrtf(128), correctly rounded, without a division's branches: by the two-word reciprocal zh + zl of sqrtf(128) (Brisebarre, Muller, Raina
// 2004: division by a divisor known in advance; tests/test_host_cpu.py compares all 2^23 significands with the division). Infinities stay,
// as zl > 0; below 2^-90 a last place may differ, which no exponential sees.
MLB_HOST_DEVICE float over_sqrt128(float x) {
#ifdef __CUDA_ARCH__
    return fmaf(x, 0x1.6a09e6p-4f, __fmul_rn(x, 0x1.9fcef4p-29f));
#else
    return std::fmaf(x, 0x1.6a09e6p-4f, x * 0x1.9fcef4p-29f);
#endif
}

}  // namespace mlb
