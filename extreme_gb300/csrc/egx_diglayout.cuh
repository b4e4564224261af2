// Places of the block matrix's entries in a stored spectral point, for the
// tensor-core contractions of the packed layout. Host and device.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define EGX_DIG_HD __host__ __device__ __forceinline__
#else
#define EGX_DIG_HD inline
#endif

namespace egx {

// The 3nz x 3nz matrix of a stored point with each component's rows and
// columns padded to an even count np: row = component * np + layer. Places in
// the packed block (GreenDims) of the entries (r, c) and (r, c + 1), c even;
// turned: entries of xz, yz, of which the staged matrix has -i times. Padded
// rows and columns name an entry beside them (of the same row, if it is a
// column), so that every place is one of the block's own. Places have 14 bits.
struct DigPair {
    int at[2];
    bool turned;
};

EGX_DIG_HD DigPair dig_pair(int nz, int r, int c) {
    const int np = (nz + 1) & ~1, S = nz * (nz + 1) / 2, lda = nz + 1, A = nz * lda;
    DigPair d;
    d.turned = false;
    for (int j = 0; j < 2; j++) {
        int cr = r / np, cc = c / np, ir = r - cr * np, ic = c - cc * np + j;
        if (ir == nz) ir--;
        if (ic == nz) ic--;
        if (cr > 2) cr = ir = 0;
        if (cc > 2) cc = ic = 0;
        d.turned = (cr == 2) != (cc == 2);
        const int lo = ir < ic ? ir : ic, hi = ir < ic ? ic : ir;
        d.at[j] = d.turned ? 4 * S + (cr == 2 ? cc * A + ic * lda + ir : cr * A + ir * lda + ic)
                           : (cr == 2 ? 3 : cr + cc) * S + lo + hi * (hi + 1) / 2;
    }
    return d;
}

// both places in a word, the flag in bit 15
EGX_DIG_HD uint32_t dig_word(int nz, int r, int c) {
    const DigPair d = dig_pair(nz, r, c);
    return (uint32_t)d.at[0] | (uint32_t)d.at[1] << 16 | (d.turned ? 1u << 15 : 0u);
}

}  // namespace egx
