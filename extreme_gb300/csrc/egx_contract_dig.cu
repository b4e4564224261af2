// Block contraction of the CIE operator (ConvolutionOperator.ApplyGreenTensorAlongZ,
// ConvolutionOperator.cs:274-327) with error-free digit products on the FP16
// tensor cores, complex128.
//
// GB300 issues two FP64 FMAs per clock and SM, so the block product in FP64
// arithmetic is bound by them; its tensor cores multiply small FP16 integers
// exactly. Every operand is written as balanced base-256 digits of a
// fixed-point number (Ozaki, Ogita, Oishi and Rump, "Error-free
// transformations of matrix multiplication by using fast routines of matrix
// multiplication and its applications", Numer. Algorithms 59 (2012)): eight
// digits (62 bits) for complex128, four (30 bits) for complex64. A product of
// two digits has 14 bits and the FP32 accumulators of mma.sync m16n8k16 add
// up 2^10 of them without a rounding. The products of digits p and q with
// p + q < 8 (4) are kept, 36 (10) of them, summed exactly per level p + q,
// joined in integers and rounded once.
//
// Scales: each stored block M (3nz x 3nz) is equilibrated by powers of two,
// M' = 2^(d_i) M 2^(d_j) with every row's largest entry near 1 (k_digitise,
// once per tensor; the exponents lie beside the digits), and the right-hand
// sides carry 2^(-d_j) and one exponent c_v each. A term is then cut 2^-61
// (2^-29) below the largest entry of M' times the largest of the scaled
// right-hand side. In the operator's own scaling (sources times layer
// thickness over the square root of the conductivity) that bound is the same
// for every layer; FP64 arithmetic loses 2^-53 of each partial sum.
//
// Algebra as in egx_contract.cu: the (up to) four spectral points that share
// a stored block are right-hand sides of one matrix after the D_p sign
// flips. Its z rows hold -A^T where its z columns hold A; with D =
// diag(1, 1, i), D M D^-1 holds -iA in both places, so the staged matrix is
// symmetric and needs no signs: X_z takes a factor i, Y_z a factor -i. The
// eight columns of an MMA are the real and imaginary parts of the four
// points: [Yr | Yi] = Mr [Xr | Xi] + Mi [-Xi | Xr].
//
// The digits of M' are a copy of the tensor, made once with the exponents:
// the upper triangle of the whole matrix in tiles of 4 x 4 sub-blocks of 2 x 2
// entries; per tile, half (digits 0-3, 4-7) and plane (re, im) 16 bytes per
// sub-block, word p the digit p of its four entries in row order. complex64
// reads the first half alone. Row 2g of a 16-row tile is the MMA's row g, row
// 2g + 1 its row g + 8, so a lane's fragment of one digit is one byte permute
// per register from two words, in either orientation of the sub-block; the
// order within a tile (sub_slot) keeps the 16-byte loads free of bank
// conflicts in both. nz = 32: 79.9 KB per point against 67.6 KB of complex128
// entries.
//
// One CTA per stored point (grid-stride), two warps per 16-row tile: one
// multiplies the real plane, the other the imaginary one, and they join
// their integer sums. The point's digits come by one bulk copy; several CTAs
// per SM overlap one's copy, conversions and sums with another's products.
//
// Measured at 128x128x32, one right-hand side: 0.64 ms per launch, against
// 4.01 ms of the FP64 kernel (k_contract<double>, 1.2 TFLOP/s, at the FP64
// pipes' rate) and 2.53 ms for two of the double-FP32 one (1.29 here). The
// products alone need 0.29 ms (2,592 MMAs per point at 8 cycles per
// sub-partition); the rest is the phases between them. 2-norm error against
// 113-bit sums, nz = 1..48: 4e-17..2.9e-16, the FP64 kernel's 9e-17..3.4e-16.
#include <cuda_fp16.h>

#include <algorithm>
#include <cstdint>

#include "egx_operator.cuh"
#include "egx_wait.cuh"

namespace egx {

namespace {

typedef unsigned long long u64;

// NS digits in HALVES groups of four, BITS of the fixed-point numbers, the
// exponent fields' EMAX (non-finite) and NORM (2^(e - NORM) above a value of
// biased exponent e), the digits' biases in a word
template <typename T> struct Dig;
template <> struct Dig<double> {
    static constexpr int NS = 8, HALVES = 2, BITS = 62, EMAX = 2047, NORM = 1022;
    typedef u64 W;
    static constexpr W BIAS = 0x4080808080808080ull;
};
template <> struct Dig<float> {
    static constexpr int NS = 4, HALVES = 1, BITS = 30, EMAX = 255, NORM = 126;
    typedef uint32_t W;
    static constexpr W BIAS = 0x40808080u;
};

constexpr int kBadBlock = 0x7fff;  // first row exponent of a block with a non-finite entry
constexpr int kNone = -(1 << 20), kNonFinite = 1 << 20;  // exponents of a right-hand side

__device__ __forceinline__ int bexp(double x) { return (int)(((uint32_t)__double2hiint(x) >> 20) & 0x7ffu); }
__device__ __forceinline__ int bexp(float x) { return (int)((__float_as_uint(x) >> 23) & 0xffu); }

// The digits of x scaled below 2^BITS: the significand with its leading bit
// at the top, shifted right by `base - (biased exponent)` (two or more). The
// low bytes hold digit + 128, the top one digit + 64; `neg` (all ones or
// zero) negates.
__device__ __forceinline__ u64 digits(double x, int base, uint32_t neg) {
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    const int e = (int)((hi >> 20) & 0x7ffu);
    const uint32_t mh = __funnelshift_l(lo, hi, 11) & 0x7fffffffu, ml = lo << 11;
    const u64 m = ((u64)(mh | (e ? 0x80000000u : 0u)) << 32) | ml;
    u64 v;
    asm("shr.u64 %0, %1, %2;" : "=l"(v) : "l"(m), "r"((uint32_t)(base - max(e, 1))));  // 64 and more: 0
    const u64 sg = (u64)(long long)(int)((uint32_t)((int)hi >> 31) ^ neg);
    return (v ^ sg) + (Dig<double>::BIAS - sg);
}
__device__ __forceinline__ uint32_t digits(float x, int base, uint32_t neg) {
    const uint32_t u = __float_as_uint(x);
    const int e = (int)((u >> 23) & 0xffu);
    const uint32_t m = (u << 8) & 0x7fffff00u | (e ? 0x80000000u : 0u);
    uint32_t v;
    asm("shr.u32 %0, %1, %2;" : "=r"(v) : "r"(m), "r"((uint32_t)(base - max(e, 1))));  // 32 and more: 0
    const uint32_t sg = (uint32_t)((int)u >> 31) ^ neg;
    return (v ^ sg) + (Dig<float>::BIAS - sg);
}

// bytes of four digit words, transposed: word k holds byte 3 - k of a, b, c, d
__device__ __forceinline__ uint4 digit_words(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    const uint32_t ab0 = __byte_perm(a, b, 0x5140), ab1 = __byte_perm(a, b, 0x7362);
    const uint32_t cd0 = __byte_perm(c, d, 0x5140), cd1 = __byte_perm(c, d, 0x7362);
    return make_uint4(__byte_perm(ab1, cd1, 0x7632), __byte_perm(ab1, cd1, 0x5410), __byte_perm(ab0, cd0, 0x7632),
                      __byte_perm(ab0, cd0, 0x5410));
}

// two bytes of a digit word (picked by sel, 0x64 above each: 1024 + field) as
// an FP16 pair, less 1024 + the field's bias
template <int P>
__device__ __forceinline__ uint32_t digit_pair(uint32_t w, uint32_t sel) {
    const uint32_t f = __byte_perm(w, 0x64646464u, sel);
    const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&f), __float2half2_rn(P == 0 ? 1088.f : 1152.f));
    return *reinterpret_cast<const uint32_t *>(&h);
}

__device__ __forceinline__ void mma_digits(float *c, const uint32_t *a, uint2 b) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y));
}

// digits P0.. P0 + 3 of a 16 x 16 tile (two sub-blocks' words, their row
// selectors) against the digits of the right-hand sides
template <int NS, int NR, int P0>
__device__ __forceinline__ void levels(float (*acc)[NS][4], uint4 u, uint4 v, uint2 su, uint2 sv, const uint2 (*b)[NS]) {
    const uint32_t uw[4] = {u.x, u.y, u.z, u.w}, vw[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        uint32_t a[4];
        if (P0 + i == 0) {
            a[0] = digit_pair<0>(uw[i], su.x), a[1] = digit_pair<0>(uw[i], su.y);
            a[2] = digit_pair<0>(vw[i], sv.x), a[3] = digit_pair<0>(vw[i], sv.y);
        } else {
            a[0] = digit_pair<1>(uw[i], su.x), a[1] = digit_pair<1>(uw[i], su.y);
            a[2] = digit_pair<1>(vw[i], sv.x), a[3] = digit_pair<1>(vw[i], sv.y);
        }
#pragma unroll
        for (int q = 0; q < NS - P0 - i; q++)
#pragma unroll
            for (int r = 0; r < NR; r++) mma_digits(acc[r][P0 + i + q], a, b[r][q]);
    }
}

// FP16 digits from P on of (u, v) at columns 2v, 2v + 1 of a fragment row
template <int NS, int P, typename W>
__device__ __forceinline__ void put_digits(uint16_t *o, W u, W v) {
    if constexpr (P < NS) {
        constexpr int byte = NS - 1 - P;
        // the two fields side by side, then as a pair
        const uint32_t x = byte >= 4 ? (uint32_t)((u64)u >> 32) : (uint32_t)u;
        const uint32_t y = byte >= 4 ? (uint32_t)((u64)v >> 32) : (uint32_t)v;
        const uint32_t h = digit_pair<P>(__byte_perm(x, y, (byte & 3) * 0x11 + 0x40), 0x4140);
        o[P * 128] = (uint16_t)h;
        o[P * 128 + 16] = (uint16_t)(h >> 16);
        put_digits<NS, P + 1>(o, u, v);
    }
}

// the joined level sums of one output: hi 2^32 + lo (complex128), or lo
struct alignas(16) Sum {
    long long hi, lo;
};
__device__ __forceinline__ Sum join(const float (*acc)[4], int c, double) {
    int s[8];
#pragma unroll
    for (int l = 0; l < 8; l++) s[l] = __float2int_rn(acc[l][c]);
    // the levels' bounds (see contract_dig_fits): 256 s0 + s1 and 256 s2 + s3 fit 32 bits
    const long long hi = (long long)(s[0] * 256 + s[1]) * 65536 + (s[2] * 256 + s[3]);
    const long long x = (long long)s[4] * 256 + s[5], y = (long long)s[6] * 256 + s[7];
    return Sum{hi, x * 65536 + y};
}
__device__ __forceinline__ Sum join(const float (*acc)[4], int c, float) {
    int s[4];
#pragma unroll
    for (int l = 0; l < 4; l++) s[l] = __float2int_rn(acc[l][c]);
    return Sum{0, (long long)(s[0] * 256 + s[1]) * 65536 + (s[2] * 256 + s[3])};
}

// the other part's share of a sum, as it is handed over
__device__ __forceinline__ void put_sum(Sum &o, Sum s) { *reinterpret_cast<longlong2 *>(&o) = make_longlong2(s.hi, s.lo); }
__device__ __forceinline__ void put_sum(long long &o, Sum s) { o = s.lo; }
__device__ __forceinline__ void add_sum(Sum &s, const Sum &o) {
    const longlong2 p = *reinterpret_cast<const longlong2 *>(&o);
    s.hi += p.x, s.lo += p.y;
}
__device__ __forceinline__ void add_sum(Sum &s, const long long &o) { s.lo += o; }

// (hi 2^32 + lo) 2^e rounded to nearest, built from the bits (not on the
// FP64 pipe); results below the normal range are 0
__device__ __forceinline__ double value(Sum s, int e, double) {
    long long h = (s.hi >> 32) + (s.lo >> 63);
    u64 l = (u64)s.hi << 32;
    l += (u64)s.lo;
    h += l < (u64)s.lo ? 1 : 0;
    const bool neg = h < 0;
    if (neg) {
        l = ~l + 1;
        h = ~h + (l == 0 ? 1 : 0);
    }
    // the top 64 bits, leading bit at bit 63, times 2^p
    u64 m;
    int p;
    if (h) {
        p = 64 - __clzll(h);
        m = ((u64)h << (64 - p)) | (l >> p);
    } else {
        if (!l) return 0.0;
        p = -__clzll((long long)l);
        m = l << -p;
    }
    m += 0x3ffull + ((m >> 11) & 1);  // to 53 bits, ties to even
    const bool carry = m < 0x8000000000000000ull;
    const int be = 1023 + 63 + p + e + (carry ? 1 : 0);
    if (be <= 0) return 0.0;
    const u64 bits =
        be >= 2047 ? 0x7ff0000000000000ull : ((u64)be << 52) | (carry ? 0 : ((m >> 11) & 0xfffffffffffffull));
    return __longlong_as_double((long long)(bits | (neg ? 0x8000000000000000ull : 0)));
}
__device__ __forceinline__ float value(Sum s, int e, float) {
    const int k = min(max(e, -250), 250), h = k / 2;
    return __ll2float_rn(s.lo) * __int_as_float((127 + h) << 23) * __int_as_float((127 + k - h) << 23);
}

// Sizes of the digit copy and of the kernel's shared memory. Rows and columns
// are counted with nz rounded up to even (np): row = component * np + layer.
struct DigGeom {
    int np, MT;           // padded layers, 16-row tiles
    int tiles;            // 8-row tiles per side
    uint32_t half, point; // bytes of a plane's half, of a point's copy
    uint32_t o_b, bytes;  // of o_b bytes of a point, the kernel's fragments
};

// NR: right-hand sides per pass
template <typename T>
__host__ __device__ inline DigGeom dig_geom(int nz, int NR = 1) {
    DigGeom g;
    g.np = (nz + 1) & ~1;
    g.MT = (3 * g.np + 15) / 16;
    g.tiles = 2 * g.MT;
    g.half = (uint32_t)(g.tiles * (g.tiles + 1) / 2) * 256u;
    g.point = 4u * g.half;
    g.o_b = (uint32_t)(2 * Dig<T>::HALVES) * g.half;
    g.bytes = g.o_b + (uint32_t)(2 * g.MT * Dig<T>::NS * NR) * 256u;
    return g;
}

// place of sub-block (i, j) in a tile of 4 x 4: lanes (2 rows x 4 columns, or
// 4 rows x 2 columns for the transposed orientation) meet distinct banks
__host__ __device__ __forceinline__ int sub_slot(int i, int j) { return i * 4 + (j ^ (i & 2)); }

__device__ __forceinline__ void pair_sync(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

// Row exponents and digits of every stored block: d with 2^(d_i + d_j) |M_ij|
// < 1 and each row's largest entry near 1, by a few steps of symmetric
// equilibration on the exponents (each step takes half of every row's
// distance from 1; all rows move together; one thread per row).
__global__ void k_digitise(const double2 *__restrict__ G, int nz, long Q, short *__restrict__ dexp,
                           unsigned char *__restrict__ out) {
    extern __shared__ short se[];  // exponent of each stored entry
    __shared__ int d[160];         // by padded row
    __shared__ int bad, top;
    const DigGeom m = dig_geom<double>(nz);
    const int S = nz * (nz + 1) / 2, lda = nz + 1, A = nz * lda, Bs = 4 * S + 2 * A, rows = 16 * m.MT;
    constexpr int kZero = -8192, kSteps = 5;
    const int r = threadIdx.x, co = r / m.np, i = r - co * m.np;
    const bool live = co < 3 && i < nz;
    for (long q = blockIdx.x; q < Q; q += gridDim.x) {
        const double2 *g = G + q * Bs;
        if (r == 0) bad = 0, top = 0;
        __syncthreads();
        for (int e = r; e < Bs; e += blockDim.x) {
            const double2 v = g[e];
            const int b = max(bexp(v.x), bexp(v.y));
            if (b == Dig<double>::EMAX) bad = 1;
            se[e] = (short)(v.x == 0.0 && v.y == 0.0 ? kZero : max(b, 1) - 1022);  // parts below 2^se
        }
        if (r < 160) d[r] = 0;
        __syncthreads();
        for (int it = 0; it <= kSteps; it++) {  // the last pass measures
            int big = kZero;
            if (live) {
                for (int ci = 0; ci < 3; ci++) {
                    const int *dc = d + ci * m.np;
                    auto take = [&](int e, int j) { big = max(big, e == kZero ? kZero : e + dc[j]); };
                    if (co == 2 ? ci < 2 : ci == 2) {
                        const short *p = se + 4 * S + (co == 2 ? ci * A + i : co * A + i * lda);
                        const int st = co == 2 ? lda : 1;
                        for (int j = 0; j < nz; j++) take(p[j * st], j);
                    } else {
                        const short *p = se + (co == 2 ? 3 : co + ci) * S;
                        const int ti = i * (i + 1) / 2;
                        for (int j = 0; j <= i; j++) take(p[ti + j], j);
                        for (int j = i + 1, tj = j * (j + 1) / 2; j < nz; tj += ++j) take(p[tj + i], j);
                    }
                }
            }
            __syncthreads();
            if (big > kZero) {
                if (it == kSteps) atomicMax(&top, big + d[r]);
                else d[r] -= (big + d[r]) >> 1;
            }
            __syncthreads();
        }
        if (live) d[r] -= (top + 1) >> 1;
        __syncthreads();
        if (r < rows) dexp[q * rows + r] = (short)(bad ? kBadBlock : d[r]);
        uint4 *o = reinterpret_cast<uint4 *>(out + (size_t)q * m.point);
        const int subs = (int)(m.half / 16);
        for (int e = r; e < subs; e += blockDim.x) {
            const int u = e >> 4;
            int TJ = (int)((sqrtf(8.f * (float)u + 1.f) - 1.f) * 0.5f);
            TJ += (TJ + 1) * (TJ + 2) / 2 <= u ? 1 : (TJ * (TJ + 1) / 2 > u ? -1 : 0);
            const int TI = u - TJ * (TJ + 1) / 2;
            const int si = (e >> 2) & 3, sj = (e & 3) ^ (si & 2);  // sub_slot's inverse
            const int r0 = 8 * TI + 2 * si, c0 = 8 * TJ + 2 * sj;
            const int cr = r0 / m.np, cc = c0 / m.np, ir = r0 - cr * m.np, ic = c0 - cc * m.np;
            u64 re[4], im[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int ii = ir + (k >> 1), jj = ic + (k & 1);
                double2 v = make_double2(0, 0);
                int base = 1024;
                const bool asym = (cr == 2) != (cc == 2);
                if (cr < 3 && cc < 3 && ii < nz && jj < nz) {
                    v = asym ? g[4 * S + (cr == 2 ? cc * A + jj * lda + ii : cr * A + ii * lda + jj)]
                             : g[(cr == 2 ? 3 : cr + cc) * S +
                                 (ii <= jj ? ii + jj * (jj + 1) / 2 : jj + ii * (ii + 1) / 2)];
                    base -= d[r0 + (k >> 1)] + d[c0 + (k & 1)];  // |v 2^(d_i + d_j)| < 1: times 2^62
                }
                const u64 x = digits(v.x, base, 0u), y = digits(v.y, base, 0u);
                re[k] = asym ? y : x;  // -i A
                im[k] = asym ? 0x8101010101010100ull - x : y;
            }
            uint4 *w = o + e;
            w[0] = digit_words((uint32_t)(re[0] >> 32), (uint32_t)(re[1] >> 32), (uint32_t)(re[2] >> 32), (uint32_t)(re[3] >> 32));
            w[2 * subs] = digit_words((uint32_t)re[0], (uint32_t)re[1], (uint32_t)re[2], (uint32_t)re[3]);
            w[subs] = digit_words((uint32_t)(im[0] >> 32), (uint32_t)(im[1] >> 32), (uint32_t)(im[2] >> 32), (uint32_t)(im[3] >> 32));
            w[3 * subs] = digit_words((uint32_t)im[0], (uint32_t)im[1], (uint32_t)im[2], (uint32_t)im[3]);
        }
        __syncthreads();
    }
}

constexpr uint64_t kWait = 2000000000ull;

template <typename T, int NR, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB)
    k_contract_dig(C<T> *buf, const unsigned char *__restrict__ G, const short *__restrict__ dexp, const OpDims d,
                   int *err) {
    constexpr int NS = Dig<T>::NS, HV = Dig<T>::HALVES;
    typedef typename Dig<T>::W W;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int sc[2][NR][4];  // exponents of the right-hand sides, by parity of the pass
    __shared__ __align__(8) uint64_t bar;
    const DigGeom m = dig_geom<T>(d.nz, NR);
    const int nz = d.nz, R = 3 * nz, MT = m.MT, KT = m.MT, rows = 16 * MT;
    uint2 *bfr = reinterpret_cast<uint2 *>(smem + m.o_b);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int part = warp >= MT ? 1 : 0, mt = warp - part * MT;
    const int Q = (d.nx + 1) * (d.ny + 1), n1 = 2 * d.ny;
    const uint32_t sbar = (uint32_t)__cvta_generic_to_shared(&bar), sG = (uint32_t)__cvta_generic_to_shared(smem);

    if (tid < 8 * NR) (&sc[0][0][0])[tid] = kNone;
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sbar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    auto fetch = [&](int q) {  // the point's digits; one thread
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sbar), "r"(m.o_b) : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sG),
            "l"(G + (size_t)q * m.point), "r"(m.o_b), "r"(sbar)
            : "memory");
    };
    __syncthreads();
    after_previous();
    if (tid == 0 && (int)blockIdx.x < Q) fetch(blockIdx.x);

    // this thread's right-hand-side entry: point xv, row xj
    const int xv = tid & 3, xj = tid >> 2, xmx = xv >> 1, xmy = xv & 1;
    const int xc = xj / m.np, xk = xj - xc * m.np;
    const bool xrow = xc < 3 && xk < nz, xz = xc == 2;
    const uint32_t xneg = ((xc == 0 && xmx) || (xc == 1 && xmy)) ? 0xffffffffu : 0u;
    // column 2 xv, row xj of a digit's fragment
    uint16_t *const bw = reinterpret_cast<uint16_t *>(bfr) + (xj >> 4) * (NS * 128) +
                         (2 * xv * 4 + ((xj & 7) >> 1)) * 4 + ((xj >> 3) & 1) * 2 + (xj & 1);
    const int row = 16 * mt + 2 * g + part;  // the output row that this thread finishes
    const int rc = row / m.np, rk = row - rc * m.np;
    const int ymx = t >> 1, ymy = t & 1;
    const bool yflip = (rc == 0 && ymx) || (rc == 1 && ymy);
    // this part's digits; this lane's tile row and its places within a tile in
    // either orientation, with the bytes of the sub-block's rows 2g (.x) and
    // 2g + 1 (.y)
    const int subs = (int)(m.half / 16);
    const uint4 *ph = reinterpret_cast<const uint4 *>(smem) + part * subs;
    const int TI = 2 * mt + (g >> 2), TI0 = TI * (TI + 1) / 2;
    const int slot_n = sub_slot(g & 3, t), slot_t = sub_slot(t, g & 3);
    const uint2 sel_n = make_uint2(0x4140, 0x4342), sel_t = make_uint2(0x4240, 0x4341);
    // one pass ahead: the right-hand side and the exponents of a point
    auto load_x = [&](int q, int rhs) {
        const int a = q / (d.ny + 1), bq = q - a * (d.ny + 1);
        const int nkx = (a == 0 || a == d.nx) ? 1 : 2;
        const int nky = (bq == 0 || bq == d.ny) ? 1 : 2;
        if (!xrow || xmx >= nkx || xmy >= nky || rhs >= d.nrhs) return mk<T>(0, 0);
        const long pt = (long)(xmx ? 2 * d.nx - a : a) * n1 + (xmy ? 2 * d.ny - bq : bq);
        return buf[pt * d.B + rhs * R + xc * nz + xk];
    };
    C<T> xnext[NR];
#pragma unroll
    for (int r = 0; r < NR; r++) xnext[r] = mk<T>(0, 0);
    int dj_next = 0, dr_next = 0, d0_next = 0;
    auto load_d = [&](int q) {
        const short *dq = dexp + (size_t)q * rows;
        dj_next = dq[xj], dr_next = dq[row], d0_next = dq[0];
    };
    if ((int)blockIdx.x < Q) {
#pragma unroll
        for (int r = 0; r < NR; r++) xnext[r] = load_x(blockIdx.x, r);
        load_d(blockIdx.x);
    }
    int pass = 0;
    uint32_t phase = 0;
    for (int q = blockIdx.x; q < Q; q += gridDim.x) {
        const int a = q / (d.ny + 1), bq = q - a * (d.ny + 1);
        const int nkx = (a == 0 || a == d.nx) ? 1 : 2;
        const int nky = (bq == 0 || bq == d.ny) ? 1 : 2;
        const int dj = dj_next, drow = dr_next, d0 = d0_next;
        bool late = false;
        for (int rhs = 0; rhs < d.nrhs; rhs += NR, pass ^= 1) {
#pragma unroll
            for (int r = 0; r < NR; r++) {
                const int xe = max(bexp(xnext[r].x), bexp(xnext[r].y));
                int cmax = xe == Dig<T>::EMAX ? kNonFinite : (xe > 0 ? xe - dj : kNone);
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) cmax = max(cmax, __shfl_xor_sync(0xffffffffu, cmax, o));
                if (lane < 4) atomicMax(&sc[pass][r][lane], cmax);
            }
            __syncthreads();
#pragma unroll
            for (int r = 0; r < NR; r++) {
                // |x 2^-dj| < 2^(c - NORM): times 2^(BITS + NORM - c)
                const C<T> x = xnext[r];
                const int base = 2 + sc[pass][r][xv] + dj;
                // X_z takes the factor i: (re, im) -> (-im, re)
                const W wr = digits(xz ? x.y : x.x, base, xneg ^ (xz ? 0xffffffffu : 0u));
                const W wi = digits(xz ? x.x : x.y, base, xneg);
                uint16_t *o = bw + r * (2 * KT * NS * 128);
                put_digits<NS, 0>(o, wr, wi);
                put_digits<NS, 0>(o + KT * (NS * 128), 2 * Dig<T>::BIAS - wi, wr);
            }
            if (rhs == 0) {
                late = !mbar_wait_ns(sbar, phase, kWait);
                if (__syncthreads_or(late)) {  // the copy did not complete in time: give up
                    if (tid == 0) {
                        atomicExch(err, EGX_ERR_TIMEOUT);
                        mbar_wait_ns(sbar, phase, kWait);
                    }
                    __syncthreads();
                    return;
                }
                phase ^= 1u;
            } else {
                __syncthreads();
            }
            if (tid < 4 * NR) (&sc[pass ^ 1][0][0])[tid] = kNone;
            // the next pass's loads, and the next point's digits on their way into
            // L2, while this one's are multiplied
            if (rhs + NR < d.nrhs) {
#pragma unroll
                for (int r = 0; r < NR; r++) xnext[r] = load_x(q, rhs + NR + r);
            } else if (q + (int)gridDim.x < Q) {
#pragma unroll
                for (int r = 0; r < NR; r++) xnext[r] = load_x(q + gridDim.x, r);
                load_d(q + gridDim.x);
                if (tid == 0)
                    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(G + (size_t)(q + gridDim.x) * m.point),
                                 "r"(m.o_b)
                                 : "memory");
            }

            float acc[NR][NS][4];
#pragma unroll
            for (int i = 0; i < NR * NS * 4; i++) (&acc[0][0][0])[i] = 0.f;
            const uint2 *bp = bfr + part * KT * (NS * 32) + lane;
            int TJ0 = 0;  // TJ (TJ + 1) / 2
#pragma unroll 1
            for (int kt = 0; kt < KT; kt++) {
                const int TJ = 2 * kt;
                const bool n0 = TI <= TJ, n1 = TI <= TJ + 1;
                const int i0 = n0 ? (TI + TJ0) * 16 + slot_n : (TJ + TI0) * 16 + slot_t;
                const int i1 = n1 ? (TI + TJ0 + TJ + 1) * 16 + slot_n : (TJ + 1 + TI0) * 16 + slot_t;
                TJ0 += 2 * TJ + 3;
                const uint2 s0 = n0 ? sel_n : sel_t, s1 = n1 ? sel_n : sel_t;
                uint2 b[NR][NS];
#pragma unroll
                for (int r = 0; r < NR; r++)
#pragma unroll
                    for (int p = 0; p < NS; p++) b[r][p] = bp[((2 * r * KT + kt) * NS + p) * 32];
                levels<NS, NR, 0>(acc, ph[i0], ph[i1], s0, s1, b);
                if constexpr (HV > 1) levels<NS, NR, 4>(acc, ph[2 * subs + i0], ph[2 * subs + i1], s0, s1, b);
            }
            __syncthreads();  // the fragments and digits are read
            if (tid == 0 && rhs + NR >= d.nrhs && q + (int)gridDim.x < Q) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                fetch(q + gridDim.x);
            }
            // the two parts meet: part 0 finishes row 2g, part 1 row 2g + 1
            typedef typename std::conditional<(HV > 1), Sum, long long>::type X;
            X *xch = reinterpret_cast<X *>(bfr);
            Sum own[NR][2];
#pragma unroll
            for (int r = 0; r < NR; r++)
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    const Sum lo = join(acc[r], c, T(0)), hi = join(acc[r], 2 + c, T(0));
                    own[r][c] = part ? hi : lo;
                    put_sum(xch[((warp * NR + r) * 2 + c) * 32 + lane], part ? lo : hi);
                }
            pair_sync(1 + mt);
            if (rc < 3 && rk < nz && ymx < nkx && ymy < nky) {
                const int cw = part ? mt : mt + MT;
#pragma unroll
                for (int r = 0; r < NR; r++) {
                    if (NR > 1 && rhs + r >= d.nrhs) break;
                    const int ct = sc[pass][r][t];
                    T y[2];
#pragma unroll
                    for (int c = 0; c < 2; c++) {
                        add_sum(own[r][c], xch[((cw * NR + r) * 2 + c) * 32 + lane]);
                        // the sides' units 2^-BITS and 2^(c - NORM - BITS), the
                        // kept levels from 256^(NS - 1) up
                        y[c] = value(own[r][c], ct - Dig<T>::NORM - 2 * Dig<T>::BITS + 8 * (NS - 1) - drow, T(0));
                    }
                    if (ct >= kNonFinite / 2 || d0 == kBadBlock) y[0] = y[1] = T(NAN);
                    // Y_z takes the factor -i: (re, im) -> (im, -re)
                    C<T> o = rc == 2 ? mk<T>(y[1], -y[0]) : mk<T>(y[0], y[1]);
                    if (yflip) o = mk<T>(-o.x, -o.y);
                    const long pt = (long)(ymx ? 2 * d.nx - a : a) * n1 + (ymy ? 2 * d.ny - bq : bq);
                    buf[pt * d.B + (rhs + r) * R + rc * nz + rk] = o;
                }
            }
        }
    }
}

template <typename T, int NR, int MAXT, int MINB>
void launch(C<T> *buf, const unsigned char *G, const short *dexp, const OpDims &d, int *err, cudaStream_t s) {
    static const int nsm = [] {
        int n = 0;
        EGX_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, 0));
        return n;
    }();
    const DigGeom m = dig_geom<T>(d.nz, NR);
    raise_smem_limit((const void *)k_contract_dig<T, NR, MAXT, MINB>, m.bytes);
    const int thr = 64 * m.MT;
    int per = 0;
    EGX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_contract_dig<T, NR, MAXT, MINB>, thr, m.bytes));
    const long Q = (long)(d.nx + 1) * (d.ny + 1);
    launch_after(buffer_bytes<T>(d), k_contract_dig<T, NR, MAXT, MINB>, (unsigned)std::min<long>(Q, (long)nsm * std::max(1, per)), thr,
                 m.bytes, s, buf, G, dexp, d, err);
}

}  // namespace

// Exact level sums: 16 x (column tiles) x (2 x 64 x 128 + 6 x 128^2) <= 2^24
// for nine tiles; digits and fragments in shared memory.
bool contract_dig_fits(int nz) {
    const DigGeom m = dig_geom<double>(nz);
    return m.MT <= 9 && m.bytes <= 226 * 1024;
}

// the digits first, the exponents behind them
static size_t digit_bytes(const GreenDims &gd) { return (size_t)gd.Q() * dig_geom<double>(gd.nz).point; }

size_t contract_dig_bytes(const GreenDims &gd) {
    return digit_bytes(gd) + (size_t)gd.Q() * 16 * dig_geom<double>(gd.nz).MT * sizeof(short);
}

void digitise(const double2 *g64, void *out, const GreenDims &gd, cudaStream_t s, long *launches) {
    const int thr = (16 * dig_geom<double>(gd.nz).MT + 31) / 32 * 32;
    unsigned char *o = static_cast<unsigned char *>(out);
    k_digitise<<<(unsigned)std::min<long>(gd.Q(), 152L * 16), thr, (size_t)gd.Bs() * sizeof(short), s>>>(
        g64, gd.nz, gd.Q(), reinterpret_cast<short *>(o + digit_bytes(gd)), o);
    EGX_CUDA(cudaGetLastError());
    if (launches) ++*launches;
}

template <typename T>
void launch_contract_dig(C<T> *buf, const void *dig, const OpDims &d, int *err, cudaStream_t s) {
    const unsigned char *G = static_cast<const unsigned char *>(dig);
    const short *dexp = reinterpret_cast<const short *>(G + digit_bytes(GreenDims{d.nx, d.ny, d.nz}));
    const int MT = dig_geom<T>(d.nz).MT;
    if (MT <= 6) launch<T, 1, 384, 2>(buf, G, dexp, d, err, s);
    else launch<T, 1, 576, 1>(buf, G, dexp, d, err, s);
}
template void launch_contract_dig<double>(double2 *, const void *, const OpDims &, int *, cudaStream_t);

}  // namespace egx
