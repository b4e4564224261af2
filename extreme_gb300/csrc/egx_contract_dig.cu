// complex128 block contraction of the CIE operator
// (ConvolutionOperator.ApplyGreenTensorAlongZ, ConvolutionOperator.cs:274-327)
// with error-free digit products on the FP16 tensor cores.
//
// GB300 issues two FP64 FMAs per clock and SM, so the block product in FP64
// arithmetic is bound by them; its tensor cores multiply small FP16 integers
// exactly. Every operand is written as eight balanced base-256 digits of a
// 62-bit fixed-point number (Ozaki, Ogita, Oishi and Rump, "Error-free
// transformations of matrix multiplication by using fast routines of matrix
// multiplication and its applications", Numer. Algorithms 59 (2012)). A product
// of two digits has 14 bits and the FP32 accumulators of mma.sync m16n8k16 add
// up 2^10 of them without a rounding. The products of digits p and q with
// p + q < 8 are kept, 36 of them, summed exactly per level p + q, joined in
// integers and rounded once.
//
// Scales. A row of the result may be many decades smaller than another (the
// tensor falls exponentially with the distance of two layers, a source may lie
// in one of them), and is as accurate all the same: the right-hand side's
// entry j is cut 62 bits below 2^(e_j), its largest over the four spectral
// points, and the matrix entry M_ij 62 bits below 2^(r_i - e_j), 2^(r_i) the
// largest |M_ij| 2^(e_j) of row i. So row i is short of the exact sum by some
// 2^-58 of its own largest term, the largest over the four points, which the
// transform back mixes. The digits of the matrix therefore depend on the
// right-hand side and are cut anew for each, from the tensor as it is stored.
//
// Algebra as in egx_contract.cu: the (up to) four spectral points that share
// a stored block are right-hand sides of one matrix after the D_p sign
// flips. Its z rows hold -A^T where its z columns hold A; with D =
// diag(1, 1, i), D M D^-1 holds -iA in both places, so the staged matrix is
// symmetric and needs no signs: X_z takes a factor i, Y_z a factor -i. The
// eight columns of an MMA are the real and imaginary parts of the four
// points: [Yr | Yi] = Mr [Xr | Xi] + Mi [-Xi | Xr].
//
// One CTA per stored point (grid-stride), two warps per 16-row tile: one
// multiplies the real plane, the other the imaginary one, and they join their
// integer sums. The point's block comes by one bulk copy. A lane takes its
// entries of a tile from the places in a table (egx_diglayout.cuh), two
// neighbouring columns of a row at a time (rows g and g + 8: the 8-byte loads
// then meet four wavefronts, their least, in every part of the packed block),
// cuts the magnitudes into digits and gives the digits their signs on the way
// to FP16.
//
// Measured at 128x128x32: 1.03 ms per launch and right-hand side, against
// 4.01 ms of the FP64 kernel (k_contract<double>, at the FP64 pipes' rate) and
// 2.53 ms for two of the double-FP32 one. Of these 0.70 are the tensor
// products, 2,592 per point, and the fragments made for them (the products
// alone need 0.29; an MMA issued between integer and FP16 instructions takes
// 11 to 18 cycles of a sub-partition instead of 8), 0.13 the row exponents. Half
// the issue slots are filled, ALU 54 %, shared memory 51 %, DRAM 16 %
// (64x64x32). 2-norm error of an apply against 64 bits 6.5e-17, the FP64
// kernel's 7.4e-17.
#include <cuda_fp16.h>

#include <algorithm>
#include <cstdint>

#include "egx_diglayout.cuh"
#include "egx_operator.cuh"
#include "egx_round.cuh"
#include "egx_wait.cuh"

namespace egx {

namespace {

typedef unsigned long long u64;

// NS digits of BITS-bit fixed-point numbers, their biases in a word; the
// exponent of non-finite values, and NORM: 2^(e - NORM) lies above a value of
// biased exponent e
constexpr int NS = 8, BITS = 62, EMAX = 2047, NORM = 1022;
constexpr u64 BIAS = 0x4080808080808080ull;

constexpr int kNone = -(1 << 20), kNonFinite = 1 << 20;  // exponents: of nothing, of a row with a non-finite entry

__device__ __forceinline__ int bexp(double x) { return (int)(((uint32_t)__double2hiint(x) >> 20) & 0x7ffu); }

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
    return (v ^ sg) + (BIAS - sg);
}

// The same of the magnitude of (hi, lo), whose exponent is not 0 or whose
// shift is 64 or more: without the significand's special case and the sign, by
// 32-bit shifts that stop at 32 (integer logic is what bounds the kernel).
__device__ __forceinline__ u64 magnitude_digits(uint32_t hi, uint32_t lo, uint32_t sh) {
    const uint32_t mh = __funnelshift_l(lo, hi, 11) | 0x80000000u, ml = lo << 11;
    const uint32_t t = __funnelshift_rc(ml, mh, sh);
    uint32_t vh, vl;
    asm("shr.u32 %0, %1, %2;" : "=r"(vh) : "r"(mh), "r"(sh));
    asm("shr.u32 %0, %1, %2;" : "=r"(vl) : "r"(t), "r"((uint32_t)max((int)sh - 32, 0)));
    return (((u64)vh << 32) | vl) + BIAS;
}

// two bytes of a word, picked by sel, with 0x64 above each: 1024 + field, FP16
__device__ __forceinline__ __half2 fields(uint32_t w, uint32_t sel) {
    const uint32_t f = __byte_perm(w, 0x64646464u, sel);
    return *reinterpret_cast<const __half2 *>(&f);
}
__device__ __forceinline__ uint32_t bits(__half2 h) { return *reinterpret_cast<const uint32_t *>(&h); }
// 1024 + the bias of digit P
template <int P> __device__ __forceinline__ __half2 offset() { return __float2half2_rn(P == 0 ? 1088.f : 1152.f); }

__device__ __forceinline__ void mma_digits(float *c, const uint32_t *a, uint2 b) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y));
}

template <int P> __device__ __forceinline__ uint32_t digit_word(u64 w) { return (uint32_t)(P < 4 ? w >> 32 : w); }

// digits P + 1 and P, then those before them, of a 16 x 16 tile (its eight
// entries' magnitudes in the fragment's order, the columns' pairs together, and
// the pairs' signs, 1 or -1) against the digits of the right-hand side at bp,
// which are read as they are needed
template <int P>
__device__ __forceinline__ void levels(float (*acc)[4], const u64 *w, const __half2 *sgn, uint2 *b, const uint2 *bp) {
    b[NS - P - 2] = bp[(NS - P - 2) * 32], b[NS - P - 1] = bp[(NS - P - 1) * 32];
    uint32_t a[2][4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        // bytes 3, 2 (P a multiple of 4) or 1, 0 of a pair's words, interleaved
        const uint32_t x = __byte_perm(digit_word<P>(w[2 * k]), digit_word<P>(w[2 * k + 1]), P % 4 ? 0x5140 : 0x7362);
        a[0][k] = bits(__hfma2(fields(x, 0x4342), sgn[k], __hneg2(__hmul2(sgn[k], offset<P>()))));
        a[1][k] = bits(__hfma2(fields(x, 0x4140), sgn[k], __hneg2(__hmul2(sgn[k], offset<P + 1>()))));
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int q = 0; q < NS - P - i; q++) mma_digits(acc[P + i + q], a[i], b[q]);
    if constexpr (P > 0) levels<P - 2>(acc, w, sgn, b, bp);
}

// FP16 digits from P on of (u, v) at columns 2v, 2v + 1 of a fragment row
template <int P>
__device__ __forceinline__ void put_digits(uint16_t *o, u64 u, u64 v) {
    if constexpr (P < NS) {
        constexpr int byte = NS - 1 - P;
        // the two fields side by side, then as a pair
        const uint32_t h = bits(__hsub2(
            fields(__byte_perm(digit_word<P>(u), digit_word<P>(v), (byte & 3) * 0x11 + 0x40), 0x4140), offset<P>()));
        o[P * 128] = (uint16_t)h;
        o[P * 128 + 16] = (uint16_t)(h >> 16);
        put_digits<P + 1>(o, u, v);
    }
}

// the joined level sums of one output: hi 2^32 + lo
struct alignas(16) Sum {
    long long hi, lo;
};
__device__ __forceinline__ Sum join(const float (*acc)[4], int c) {
    int s[8];
#pragma unroll
    for (int l = 0; l < 8; l++) s[l] = __float2int_rn(acc[l][c]);
    // the levels' bounds (see contract_dig_fits): 256 s0 + s1 and 256 s2 + s3 fit 32 bits
    const long long hi = (long long)(s[0] * 256 + s[1]) * 65536 + (s[2] * 256 + s[3]);
    const long long x = (long long)s[4] * 256 + s[5], y = (long long)s[6] * 256 + s[7];
    return Sum{hi, x * 65536 + y};
}

// (hi 2^32 + lo) 2^e rounded to nearest, built from the bits (not on the FP64
// pipe)
__device__ __forceinline__ double value(Sum s, int e) {
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
    return round_f64(m, p + e, neg ? 0x80000000u : 0u);
}

// The kernel's shared memory. Rows and columns are counted with nz rounded up
// to even (np): row = component * np + layer.
struct DigGeom {
    int np, MT;              // padded layers, 16-row tiles
    uint32_t point;          // bytes of a point's block
    uint32_t o_b, o_tab;     // fragments of the right-hand side, places of the sub-blocks
    uint32_t o_e, o_r, bytes;  // exponents by column, by row and part
};

__host__ __device__ inline DigGeom dig_geom(int nz) {
    DigGeom g;
    g.np = (nz + 1) & ~1;
    g.MT = (3 * g.np + 15) / 16;
    g.point = (uint32_t)(4 * nz * (nz + 1)) * (uint32_t)sizeof(double2);
    g.o_b = g.point;
    g.o_tab = g.o_b + (uint32_t)(2 * g.MT * NS) * 256u;
    g.o_e = g.o_tab + (uint32_t)(g.MT * g.MT) * 512u;
    g.o_r = g.o_e + (uint32_t)g.MT * 64u;
    g.bytes = g.o_r + (uint32_t)g.MT * 128u;
    return g;
}

__device__ __forceinline__ void pair_sync(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

constexpr int kFloor = 66;
constexpr uint64_t kWait = 2000000000ull;

template <int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB)
    k_contract_dig(double2 *buf, const double2 *__restrict__ G, const OpDims d, int *err) {
    extern __shared__ __align__(128) unsigned char smem[];
    // by parity of the pass: points with a non-finite right-hand side, the largest exponent
    __shared__ int bad[2][4], emax[2];
    __shared__ __align__(8) uint64_t bar;
    const DigGeom m = dig_geom(d.nz);
    const int nz = d.nz, R = 3 * nz, MT = m.MT, KT = m.MT;
    uint2 *bfr = reinterpret_cast<uint2 *>(smem + m.o_b);
    uint4 *tab = reinterpret_cast<uint4 *>(smem + m.o_tab);
    int *se = reinterpret_cast<int *>(smem + m.o_e), *sr = reinterpret_cast<int *>(smem + m.o_r);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int part = warp >= MT ? 1 : 0, mt = warp - part * MT;
    const int Q = (d.nx + 1) * (d.ny + 1), n1 = 2 * d.ny;
    const uint32_t sbar = (uint32_t)__cvta_generic_to_shared(&bar), sG = (uint32_t)__cvta_generic_to_shared(smem);

    if (tid < 8) (&bad[0][0])[tid] = 0;
    if (tid < 2) emax[tid] = kNone;
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sbar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // a lane's entries of a tile: rows g and g + 8, columns 2t, 2t + 1 and 8 on
    for (int i = tid; i < MT * KT * 32; i += blockDim.x) {
        const int ln = i & 31, tile = i >> 5, tm = tile / KT, r = 16 * tm + (ln >> 2);
        const int c = 16 * (tile - tm * KT) + 2 * (ln & 3);
        tab[i] = make_uint4(dig_word(nz, r, c), dig_word(nz, r + 8, c), dig_word(nz, r, c + 8),
                            dig_word(nz, r + 8, c + 8));
    }
    auto fetch = [&](int q) {  // the point's block; one thread
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sbar), "r"(m.point) : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sG),
            "l"(reinterpret_cast<const unsigned char *>(G) + (size_t)q * m.point), "r"(m.point), "r"(sbar)
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
    const int row = 16 * mt + g + 8 * part;  // the output row that this thread finishes
    const int rc = row / m.np, rk = row - rc * m.np;
    const int ymx = t >> 1, ymy = t & 1;
    const bool yflip = (rc == 0 && ymx) || (rc == 1 && ymy);
    const uint4 *const tab_l = tab + mt * KT * 32 + lane;
    const int2 *const se_l = reinterpret_cast<const int2 *>(se) + t;
    // one pass ahead: the right-hand side of a point
    auto load_x = [&](int q, int rhs) {
        const int a = q / (d.ny + 1), bq = q - a * (d.ny + 1);
        const int nkx = (a == 0 || a == d.nx) ? 1 : 2;
        const int nky = (bq == 0 || bq == d.ny) ? 1 : 2;
        if (!xrow || xmx >= nkx || xmy >= nky) return make_double2(0, 0);
        const long pt = (long)(xmx ? 2 * d.nx - a : a) * n1 + (xmy ? 2 * d.ny - bq : bq);
        return buf[pt * d.B + rhs * R + xc * nz + xk];
    };
    double2 xnext = make_double2(0, 0);
    if ((int)blockIdx.x < Q) xnext = load_x(blockIdx.x, 0);
    int pass = 0;
    uint32_t phase = 0;
    for (int q = blockIdx.x; q < Q; q += gridDim.x) {
        const int a = q / (d.ny + 1), bq = q - a * (d.ny + 1);
        const int nkx = (a == 0 || a == d.nx) ? 1 : 2;
        const int nky = (bq == 0 || bq == d.ny) ? 1 : 2;
        bool late = false;
        for (int rhs = 0; rhs < d.nrhs; rhs++, pass ^= 1) {
            const double2 x = xnext;
            int ex = x.x == 0.0 && x.y == 0.0 ? kNone : max(max(bexp(x.x), bexp(x.y)), 1);
            if (ex == EMAX) {
                bad[pass][xv] = 1;
                ex = kNone;
            }
            ex = max(ex, __shfl_xor_sync(0xffffffffu, ex, 1));
            ex = max(ex, __shfl_xor_sync(0xffffffffu, ex, 2));
            const int et = __reduce_max_sync(0xffffffffu, ex);
            if (lane == 0) atomicMax(&emax[pass], et);
            __syncthreads();  // the last pass's sums and exponents are read
            if (xv == 0) se[xj] = ex;
            {
                // |x| < 2^(ex - NORM): times 2^(BITS + NORM - ex). X_z takes the
                // factor i: (re, im) -> (-im, re)
                const u64 wr = digits(xz ? x.y : x.x, 2 + ex, xneg ^ (xz ? 0xffffffffu : 0u));
                const u64 wi = digits(xz ? x.x : x.y, 2 + ex, xneg);
                put_digits<0>(bw, wr, wi);
                put_digits<0>(bw + KT * (NS * 128), 2 * BIAS - wi, wr);
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
            if (tid < 4) bad[pass ^ 1][tid] = 0;
            if (tid == 0) emax[pass ^ 1] = kNone;
            // the next pass's loads, and the next point's block on its way into
            // L2, while this one is multiplied
            if (rhs + 1 < d.nrhs) {
                xnext = load_x(q, rhs + 1);
            } else if (q + (int)gridDim.x < Q) {
                xnext = load_x(q + gridDim.x, 0);
                if (tid == 0)
                    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(
                                     reinterpret_cast<const unsigned char *>(G) + (size_t)(q + gridDim.x) * m.point),
                                 "r"(m.point)
                                 : "memory");
            }

            // The rows' exponents, each part over its half of the column tiles:
            // the high words' magnitudes plus 2^20 (e_j - the largest e). At
            // least kFloor above it, so that zeros and entries below 2^-1022
            // are shifted out; a row is short of its terms where they all lie
            // below 2^(kFloor - 1022) of the largest right-hand side.
            int r0, r1;
            {
                const int top = emax[pass];
                int m0 = kFloor << 20, m1 = m0;
                uint32_t big0 = 0, big1 = 0;
                const uint4 *M = reinterpret_cast<const uint4 *>(smem);
                for (int kt = part; kt < KT; kt += 2) {
                    const uint4 w = tab_l[kt * 32];
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const uint32_t w0 = h ? w.z : w.x, w1 = h ? w.w : w.y;
                        const int2 e = se_l[8 * kt + 4 * h];
                        const int ex = max(e.x - top, -2047) << 20, ey = max(e.y - top, -2047) << 20;
                        auto high = [&](uint32_t at) {
                            const uint4 z = M[at];
                            return max(z.y & 0x7fffffffu, z.w & 0x7fffffffu);
                        };
                        const uint32_t h00 = high(w0 & 0x3fffu), h01 = high(w0 >> 16);
                        const uint32_t h10 = high(w1 & 0x3fffu), h11 = high(w1 >> 16);
                        m0 = max(m0, max((int)h00 + ex, (int)h01 + ey));
                        m1 = max(m1, max((int)h10 + ex, (int)h11 + ey));
                        big0 = max(big0, max(h00, h01));
                        big1 = max(big1, max(h10, h11));
                    }
                }
                r0 = big0 >= 0x7ff00000u ? kNonFinite : (m0 >> 20) + top;
                r1 = big1 >= 0x7ff00000u ? kNonFinite : (m1 >> 20) + top;
#pragma unroll
                for (int o = 1; o < 4; o <<= 1) {
                    r0 = max(r0, __shfl_xor_sync(0xffffffffu, r0, o));
                    r1 = max(r1, __shfl_xor_sync(0xffffffffu, r1, o));
                }
                int2 *rp = reinterpret_cast<int2 *>(sr) + mt * 8 + g;
                if (t == 0) rp[part * 8 * MT] = make_int2(r0, r1);
                pair_sync(1 + mt);
                const int2 o = rp[(part ^ 1) * 8 * MT];
                r0 = max(r0, o.x), r1 = max(r1, o.y);
            }

            float acc[NS][4];
#pragma unroll
            for (int i = 0; i < NS * 4; i++) (&acc[0][0])[i] = 0.f;
            const uint2 *bp = bfr + part * KT * (NS * 32) + lane;
            // this plane's words of the block; of turned entries -i (re, im) =
            // (im, -re): the other plane's, and the real one's with the sign
            const unsigned char *const plane = smem + 8 * part;
            const int other = part ? -1 : 1;
            const uint32_t flip = part ? 0x10001000u : 0u;
#pragma unroll 1
            for (int kt = 0; kt < KT; kt++) {
                const uint4 w = tab_l[kt * 32];
                u64 dw[8];  // rows g, g + 8 of the first columns, of the second
                __half2 sgn[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const uint32_t wk = k == 0 ? w.x : k == 1 ? w.y : k == 2 ? w.z : w.w;
                    const int2 e = se_l[8 * kt + 4 * (k >> 1)];
                    const int r = 2 + (k & 1 ? r1 : r0);
                    const uint32_t turned = (wk & 0x8000u) >> 12;  // 8 or 0
                    const unsigned char *p = plane + other * (int)turned;
                    const uint2 u = *reinterpret_cast<const uint2 *>(p + (wk & 0x3fffu) * 16u);
                    const uint2 v = *reinterpret_cast<const uint2 *>(p + (wk >> 16) * 16u);
                    dw[2 * k] = magnitude_digits(u.y, u.x, (uint32_t)(r - e.x - (int)((u.y + u.y) >> 21)));
                    dw[2 * k + 1] = magnitude_digits(v.y, v.x, (uint32_t)(r - e.y - (int)((v.y + v.y) >> 21)));
                    const uint32_t sg = (__byte_perm(u.y, v.y, 0x7632) & 0x80008000u) ^ (0x3c003c00u + turned * flip);
                    sgn[k] = *reinterpret_cast<const __half2 *>(&sg);
                }
                uint2 b[NS];
                levels<NS - 2>(acc, dw, sgn, b, bp + kt * (NS * 32));
            }
            __syncthreads();  // the fragments and the block are read
            if (tid == 0 && rhs + 1 == d.nrhs && q + (int)gridDim.x < Q) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                fetch(q + gridDim.x);
            }
            // the two parts meet: part 0 finishes row g, part 1 row g + 8
            Sum *xch = reinterpret_cast<Sum *>(bfr);
            Sum own[2];
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const Sum lo = join(acc, c), hi = join(acc, 2 + c);
                own[c] = part ? hi : lo;
                xch[(warp * 2 + c) * 32 + lane] = part ? lo : hi;
            }
            const int nonfinite = bad[pass][t];
            pair_sync(1 + mt);
            if (rc < 3 && rk < nz && ymx < nkx && ymy < nky) {
                const int cw = part ? mt : mt + MT, re = part ? r1 : r0;
                double y[2];
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    const Sum o = xch[(cw * 2 + c) * 32 + lane];
                    own[c].hi += o.hi, own[c].lo += o.lo;
                    // the sides' units 2^(r - e - NORM - BITS) and 2^(e - NORM - BITS),
                    // the kept levels from 256^(NS - 1) up
                    y[c] = value(own[c], re - 2 * (NORM + BITS) + 8 * (NS - 1));
                }
                if (nonfinite || re == kNonFinite) y[0] = y[1] = (double)NAN;
                // Y_z takes the factor -i: (re, im) -> (im, -re)
                double2 o = rc == 2 ? make_double2(y[1], -y[0]) : make_double2(y[0], y[1]);
                if (yflip) o = make_double2(-o.x, -o.y);
                const long pt = (long)(ymx ? 2 * d.nx - a : a) * n1 + (ymy ? 2 * d.ny - bq : bq);
                buf[pt * d.B + rhs * R + rc * nz + rk] = o;
            }
        }
    }
}

template <int MAXT, int MINB>
void launch(double2 *buf, const double2 *G, const OpDims &d, int *err, cudaStream_t s) {
    static const int nsm = [] {
        int n = 0;
        EGX_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, 0));
        return n;
    }();
    const DigGeom m = dig_geom(d.nz);
    const auto kernel = k_contract_dig<MAXT, MINB>;
    raise_smem_limit((const void *)kernel, m.bytes);
    const int thr = 64 * m.MT;
    int per = 0;
    EGX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, thr, m.bytes));
    const long Q = (long)(d.nx + 1) * (d.ny + 1);
    const unsigned grid = (unsigned)std::min<long>(Q, (long)nsm * std::max(1, per));
    launch_after(buffer_bytes<double>(d), kernel, grid, thr, m.bytes, s, buf, G, d, err);
}

}  // namespace

// Exact level sums: 16 x (column tiles) x (2 x 64 x 128 + 6 x 128^2) <= 2^24
// for nine tiles; block and fragments in shared memory.
bool contract_dig_fits(int nz) {
    const DigGeom m = dig_geom(nz);
    return m.MT <= 9 && m.bytes <= 226 * 1024;
}

void launch_contract_dig(double2 *buf, const double2 *G, const OpDims &d, int *err, cudaStream_t s) {
    // two blocks per SM where their shared memory fits; up to five tiles with
    // more registers for it (96 instead of 80: nz = 24 560 us against 578, nz = 4
    // 103 against 115, nz = 12 321 against 316)
    const int MT = dig_geom(d.nz).MT;
    if (MT <= 5) launch<320, 2>(buf, G, d, err, s);
    else if (MT == 6) launch<384, 2>(buf, G, d, err, s);
    else launch<576, 1>(buf, G, d, err, s);
}

}  // namespace egx
