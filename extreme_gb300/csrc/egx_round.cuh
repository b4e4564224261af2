// Rounding of integers to complex128 parts, for the kernels that compute them
// on the integer pipes.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace egx {

// v 2^e as an FP64 number, v's leading bit at bit 63, with the sign bit `sign`
// of its high word: rounded to nearest, ties to even. Below the normal range a
// product by a power of two rounds once more.
__device__ __forceinline__ double round_f64(unsigned long long v, int e, uint32_t sign) {
    v += 0x3ffull + ((v >> 11) & 1);  // to 53 bits
    const bool carry = v < 0x8000000000000000ull;
    const int be = 1023 + 63 + e + (carry ? 1 : 0);
    const unsigned long long f = carry ? 0 : ((v >> 11) & 0xfffffffffffffull);
    if (be >= 2047) return __hiloint2double((int)(sign | 0x7ff00000u), 0);
    const int up = be > 0 ? be : max(be + 128, 0);
    const double r = __hiloint2double((int)(sign | ((uint32_t)up << 20) | (uint32_t)(f >> 32)), (int)(uint32_t)f);
    return be > 0 ? r : r * 2.938735877055719e-39;  // 2^-128
}

}  // namespace egx
