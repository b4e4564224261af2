// Rounding of integers to complex128 parts, for the kernels that compute them
// on the integer pipes.
#pragma once

#include <cuda_runtime.h>

namespace egx {

// m 2^e as an FP64 number with the sign of neg, rounded to nearest, ties to
// even, gradual underflow included; m's leading bit is at bit 63
__device__ __forceinline__ double round_f64(unsigned long long m, int e, bool neg) {
    const unsigned long long sign = neg ? 0x8000000000000000ull : 0;
    int be = 1023 + 63 + e;
    unsigned long long bits;
    if (be > 0) {
        m += 0x3ffull + ((m >> 11) & 1);  // to 53 bits
        const bool carry = m < 0x8000000000000000ull;
        be += carry ? 1 : 0;
        bits = be >= 2047 ? 0x7ff0000000000000ull
                          : ((unsigned long long)be << 52) | (carry ? 0 : ((m >> 11) & 0xfffffffffffffull));
    } else {  // below the normal range: bits in units of 2^-1074
        const int s = 12 - be;
        if (s > 64) return __longlong_as_double((long long)sign);
        const unsigned long long k = s < 64 ? m >> s : 0, rest = m << (64 - s);  // s >= 12
        bits = k + (rest > 0x8000000000000000ull || (rest == 0x8000000000000000ull && (k & 1)) ? 1 : 0);
    }
    return __longlong_as_double((long long)(bits | sign));
}

}  // namespace egx
