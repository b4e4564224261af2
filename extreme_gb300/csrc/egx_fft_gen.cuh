// Batched DFT of BT interleaved columns of any 7-smooth length, one CTA per
// line and tile of columns: a Stockham autosort transform (see egx_fft.cuh)
// whose first stage reads its elements from global memory into registers and
// whose last stage stores from registers, with one shared buffer [n][BT]
// between (the stages in the middle read, meet at a barrier and write).
//
// Two arithmetics:
//  * float: complex64 as it is, for the lengths without a register plan
//    (egx_fft_reg.cuh): 360-point lines of 240 x 210 columns 76 us, the
//    Stockham kernel's 214.
//  * double: every column of a line is one block-floating-point number set,
//    64-bit integers under the exponent of its largest part. GB300's FP64 pipe
//    issues two operations per clock and SM, its integer pipes 32 64-bit
//    additions and some ten 64 x 64 -> 64 high products, so a complex128
//    transform that reads and writes complex128 runs several times faster on
//    integers. Inputs lie below 2^59; a stage of radix R grows a bound of the
//    values by R, and the next one's twiddles (62 bits) take back, rounding,
//    the least whole bits (two or more) that keep its results below 2^62.85,
//    where no sum of the stage and no product of a twiddle overflows. The
//    roundings stay 2^-59 of that growing bound: by 2-norm the result's error
//    was 0.15 to 0.5 times an FP64 transform's, over all lengths and inputs
//    tried (noise, single peaks, decaying, scaled over 20 decades, zero-padded,
//    constant). A whole 256 x 256 x 96 pass takes 83 us, the FP64 register
//    transform took 330. The integer pipes bound it (256 x 256 x 48: ALU 67 %,
//    issue slots 66 %, DRAM 14 %).
//
// The inverse transform is the forward one with real and imaginary parts
// exchanged on the way in and out.
#pragma once

#include <cstdint>

#include "egx_fft.cuh"

namespace egx {

// ------------------------------------------------------------ arithmetics
struct FftFloat {
    typedef float S;
    typedef float2 V;
    typedef float2 Tw;
    static __device__ __forceinline__ V add(V a, V b) { return make_float2(a.x + b.x, a.y + b.y); }
    static __device__ __forceinline__ V sub(V a, V b) { return make_float2(a.x - b.x, a.y - b.y); }
    static __device__ __forceinline__ V mul_mi(V a) { return make_float2(a.y, -a.x); }  // -i a
    template <class K> static __device__ __forceinline__ V scale(V a) {
        return make_float2(a.x * (float)K::c, a.y * (float)K::c);
    }
    static __device__ __forceinline__ V half(V a) { return make_float2(0.5f * a.x, 0.5f * a.y); }
    static __device__ __forceinline__ V quarter(V a) { return make_float2(0.25f * a.x, 0.25f * a.y); }
    static __device__ __forceinline__ V tw(V a, Tw w, int) {
        return make_float2(a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x);
    }
    static __device__ __forceinline__ V down(V a, int) { return a; }
};

struct __align__(16) FixC {
    long long x, y;
};

struct FftFixed {
    typedef long long S;
    typedef FixC V;
    typedef int4 Tw;  // (x 2^-32 + y 2^-64, z 2^-32 + w 2^-64): the twiddle times 2^-sh
    static __device__ __forceinline__ V add(V a, V b) { return V{a.x + b.x, a.y + b.y}; }
    static __device__ __forceinline__ V sub(V a, V b) { return V{a.x - b.x, a.y - b.y}; }
    static __device__ __forceinline__ V mul_mi(V a) { return V{a.y, -a.x}; }
    // x = hi 2^32 + lo, both signed
    static __device__ __forceinline__ void split(S x, int &hi, int &lo) {
        lo = (int)(uint32_t)x;
        hi = (int)(x >> 32) + (int)((uint32_t)lo >> 31);
    }
    static __device__ __forceinline__ S mad(int a, int b, S c) { return (S)a * (S)b + c; }
    // x c, c = h 2^-31 + l 2^-63
    static __device__ __forceinline__ S mulc(S x, int h, int l) {
        int xh, xl;
        split(x, xh, xl);
        const S u = mad(xl, h, mad(xh, l, 1ll << 30));
        const S t = (S)xh * h;
        return t + t + (u >> 31);
    }
    template <class K> static __device__ __forceinline__ V scale(V a) {
        return V{mulc(a.x, K::h, K::l), mulc(a.y, K::h, K::l)};
    }
    static __device__ __forceinline__ V half(V a) { return V{(a.x + 1) >> 1, (a.y + 1) >> 1}; }
    static __device__ __forceinline__ V quarter(V a) { return V{(a.x + 2) >> 2, (a.y + 2) >> 2}; }
    static __device__ __forceinline__ V tw(V a, Tw w, int) {
        int xh, xl, yh, yl;
        split(a.x, xh, xl);
        split(a.y, yh, yl);
        const int nz = -w.z, nw = -w.w;
        const S ur = mad(xl, w.x, mad(xh, w.y, mad(yl, nz, mad(yh, nw, 1ll << 31))));
        const S ui = mad(xl, w.z, mad(xh, w.w, mad(yl, w.x, mad(yh, w.y, 1ll << 31))));
        return V{mad(xh, w.x, mad(yh, nz, ur >> 32)), mad(xh, w.z, mad(yh, w.x, ui >> 32))};
    }
    static __device__ __forceinline__ V down(V a, int sh) {
        const S r = (1ll << sh) >> 1;
        return V{(a.x + r) >> sh, (a.y + r) >> sh};
    }
};

// constants c = h 2^-31 + l 2^-63
#define EGX_FFT_CONST(name, val, hh, ll)        \
    struct name {                               \
        static constexpr double c = val;        \
        static constexpr int h = hh, l = ll;    \
    }
EGX_FFT_CONST(KHalfRoot2, 0.7071067811865476, 1518500250, -51432894);
EGX_FFT_CONST(KHalfRoot3, 0.8660254037844386, 1859775393, 1630710223);
EGX_FFT_CONST(KQuarterRoot5, 0.5590169943749475, 1200479854, 1607638789);
EGX_FFT_CONST(KSin5_1, 0.9510565162951535, 2042378317, 290717050);
EGX_FFT_CONST(KSin5_2, 0.5877852522924731, 1262259218, -714508361);
EGX_FFT_CONST(KCos7_1, 0.6234898018587335, 1338934154, 800540083);
EGX_FFT_CONST(KCos7_2, -0.2225209339563144, -477860067, -38109801);
EGX_FFT_CONST(KCos7_3, -0.9009688679024191, -1934815911, -762430282);
EGX_FFT_CONST(KSin7_1, 0.7818314824680298, 1678970324, 393817135);
EGX_FFT_CONST(KSin7_2, 0.9749279121818236, 2093641749, 1671799694);
EGX_FFT_CONST(KSin7_3, 0.4338837391175581, 931758235, -480804351);
EGX_FFT_CONST(KCos9_1, 0.766044443118978, 1645067915, 1027663049);
EGX_FFT_CONST(KSin9_1, 0.6427876096865394, 1380375881, -262638930);
EGX_FFT_CONST(KCos9_2, 0.17364817766693036, 372906622, 192121251);
EGX_FFT_CONST(KSin9_2, 0.984807753012208, 2114858546, 74472808);
EGX_FFT_CONST(KCos9_4, -0.9396926207859084, -2017974537, -1219784300);
EGX_FFT_CONST(KSin9_4, 0.3420201433256687, 734482665, 337111738);
#undef EGX_FFT_CONST

// ------------------------------------------------------------- butterflies
// forward DFTs (exp(-2 pi i k r / R)) in registers
template <class A> __device__ __forceinline__ void gdft2(typename A::V &a, typename A::V &b) {
    const typename A::V t = a;
    a = A::add(t, b);
    b = A::sub(t, b);
}
template <class A> __device__ __forceinline__ void gdft3(typename A::V &a, typename A::V &b, typename A::V &c) {
    typedef typename A::V V;
    const V t = A::add(b, c), m = A::sub(a, A::half(t)), s = A::mul_mi(A::template scale<KHalfRoot3>(A::sub(b, c)));
    a = A::add(a, t);
    b = A::add(m, s);
    c = A::sub(m, s);
}
template <class A> __device__ __forceinline__ void gdft4(typename A::V &a, typename A::V &b, typename A::V &c,
                                                         typename A::V &d) {
    typedef typename A::V V;
    const V a0 = A::add(a, c), a1 = A::sub(a, c), b0 = A::add(b, d), b1 = A::mul_mi(A::sub(b, d));
    a = A::add(a0, b0);
    c = A::sub(a0, b0);
    b = A::add(a1, b1);
    d = A::sub(a1, b1);
}
template <class A, int R> struct Gdft;
template <class A> struct Gdft<A, 2> {
    static __device__ __forceinline__ void run(typename A::V *v) { gdft2<A>(v[0], v[1]); }
};
template <class A> struct Gdft<A, 3> {
    static __device__ __forceinline__ void run(typename A::V *v) { gdft3<A>(v[0], v[1], v[2]); }
};
template <class A> struct Gdft<A, 4> {
    static __device__ __forceinline__ void run(typename A::V *v) { gdft4<A>(v[0], v[1], v[2], v[3]); }
};
template <class A> struct Gdft<A, 5> {
    static __device__ __forceinline__ void run(typename A::V *v) {
        typedef typename A::V V;
        const V t1 = A::add(v[1], v[4]), t2 = A::add(v[2], v[3]), t3 = A::sub(v[1], v[4]), t4 = A::sub(v[2], v[3]);
        const V t5 = A::add(t1, t2);
        const V m = A::sub(v[0], A::quarter(t5)), q = A::template scale<KQuarterRoot5>(A::sub(t1, t2));
        const V a = A::add(m, q), b = A::sub(m, q);
        const V c = A::mul_mi(A::add(A::template scale<KSin5_1>(t3), A::template scale<KSin5_2>(t4)));
        const V d = A::mul_mi(A::sub(A::template scale<KSin5_2>(t3), A::template scale<KSin5_1>(t4)));
        v[0] = A::add(v[0], t5);
        v[1] = A::add(a, c);
        v[4] = A::sub(a, c);
        v[2] = A::add(b, d);
        v[3] = A::sub(b, d);
    }
};
// 6 = 2 x 3, coprime: no twiddles between (Good's mapping)
template <class A> struct Gdft<A, 6> {
    static __device__ __forceinline__ void run(typename A::V *v) {
        typedef typename A::V V;
        V a0 = v[0], a1 = v[2], a2 = v[4], b0 = v[3], b1 = v[5], b2 = v[1];
        gdft3<A>(a0, a1, a2);
        gdft3<A>(b0, b1, b2);
        v[0] = A::add(a0, b0);
        v[3] = A::sub(a0, b0);
        v[4] = A::add(a1, b1);
        v[1] = A::sub(a1, b1);
        v[2] = A::add(a2, b2);
        v[5] = A::sub(a2, b2);
    }
};
template <class A> struct Gdft<A, 7> {
    static __device__ __forceinline__ void run(typename A::V *v) {
        typedef typename A::V V;
        const V p1 = A::add(v[1], v[6]), p2 = A::add(v[2], v[5]), p3 = A::add(v[3], v[4]);
        const V m1 = A::sub(v[1], v[6]), m2 = A::sub(v[2], v[5]), m3 = A::sub(v[3], v[4]);
        const V v0 = v[0];
        v[0] = A::add(A::add(v0, p1), A::add(p2, p3));
        auto even = [&](V a, V b, V c) {  // v0 + cos1 a + cos2 b + cos3 c
            return A::add(A::add(v0, A::template scale<KCos7_1>(a)),
                          A::add(A::template scale<KCos7_2>(b), A::template scale<KCos7_3>(c)));
        };
        {
            const V e = even(p1, p2, p3);
            const V o = A::mul_mi(A::add(A::add(A::template scale<KSin7_1>(m1), A::template scale<KSin7_2>(m2)),
                                         A::template scale<KSin7_3>(m3)));
            v[1] = A::add(e, o);
            v[6] = A::sub(e, o);
        }
        {
            const V e = even(p3, p1, p2);
            const V o = A::mul_mi(A::sub(A::sub(A::template scale<KSin7_2>(m1), A::template scale<KSin7_3>(m2)),
                                         A::template scale<KSin7_1>(m3)));
            v[2] = A::add(e, o);
            v[5] = A::sub(e, o);
        }
        {
            const V e = even(p2, p3, p1);
            const V o = A::mul_mi(A::add(A::sub(A::template scale<KSin7_3>(m1), A::template scale<KSin7_1>(m2)),
                                         A::template scale<KSin7_2>(m3)));
            v[3] = A::add(e, o);
            v[4] = A::sub(e, o);
        }
    }
};
template <class A> struct Gdft<A, 8> {
    static __device__ __forceinline__ void run(typename A::V *v) {
        typedef typename A::V V;
        V e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
        gdft4<A>(e0, e1, e2, e3);
        gdft4<A>(o0, o1, o2, o3);
        // o_k *= exp(-2 pi i k / 8)
        o1 = A::template scale<KHalfRoot2>(A::add(o1, A::mul_mi(o1)));
        o2 = A::mul_mi(o2);
        o3 = A::template scale<KHalfRoot2>(A::sub(A::mul_mi(o3), o3));
        v[0] = A::add(e0, o0);
        v[4] = A::sub(e0, o0);
        v[1] = A::add(e1, o1);
        v[5] = A::sub(e1, o1);
        v[2] = A::add(e2, o2);
        v[6] = A::sub(e2, o2);
        v[3] = A::add(e3, o3);
        v[7] = A::sub(e3, o3);
    }
};

// 9 = 3 x 3: n = 3 n1 + n2, k = k1 + 3 k2, twiddles W9^(n2 k1)
template <class A> struct Gdft<A, 9> {
    template <class Cs, class Sn> static __device__ __forceinline__ typename A::V rot(typename A::V a) {
        // a (cos - i sin)
        return A::add(A::template scale<Cs>(a), A::mul_mi(A::template scale<Sn>(a)));
    }
    static __device__ __forceinline__ void run(typename A::V *v) {
        typedef typename A::V V;
        V a0 = v[0], a1 = v[3], a2 = v[6], b0 = v[1], b1 = v[4], b2 = v[7], c0 = v[2], c1 = v[5], c2 = v[8];
        gdft3<A>(a0, a1, a2);
        gdft3<A>(b0, b1, b2);
        gdft3<A>(c0, c1, c2);
        b1 = rot<KCos9_1, KSin9_1>(b1);
        b2 = rot<KCos9_2, KSin9_2>(b2);
        c1 = rot<KCos9_2, KSin9_2>(c1);
        c2 = rot<KCos9_4, KSin9_4>(c2);
        gdft3<A>(a0, b0, c0);
        gdft3<A>(a1, b1, c1);
        gdft3<A>(a2, b2, c2);
        v[0] = a0, v[1] = a1, v[2] = a2, v[3] = b0, v[4] = b1, v[5] = b2, v[6] = c0, v[7] = c1, v[8] = c2;
    }
};
// 10 = 2 x 5, coprime (Good's mapping)
template <class A> struct Gdft<A, 10> {
    static __device__ __forceinline__ void run(typename A::V *v) {
        typedef typename A::V V;
        V a[5] = {v[0], v[2], v[4], v[6], v[8]}, b[5] = {v[5], v[7], v[9], v[1], v[3]};
        Gdft<A, 5>::run(a);
        Gdft<A, 5>::run(b);
        // k = 0, 6, 2, 8, 4 (even) and 5, 1, 7, 3, 9 (odd) for k mod 5 = 0..4
        v[0] = A::add(a[0], b[0]), v[5] = A::sub(a[0], b[0]);
        v[6] = A::add(a[1], b[1]), v[1] = A::sub(a[1], b[1]);
        v[2] = A::add(a[2], b[2]), v[7] = A::sub(a[2], b[2]);
        v[8] = A::add(a[3], b[3]), v[3] = A::sub(a[3], b[3]);
        v[4] = A::add(a[4], b[4]), v[9] = A::sub(a[4], b[4]);
    }
};

// ------------------------------------------------- block floating point
// x 2^(59 + 1022 - E) rounded, |x| < 2^(E - 1022)
__device__ __forceinline__ long long fix_in(double x, int E) {
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    const int e = (int)((hi >> 20) & 0x7ffu);
    const uint32_t mh = __funnelshift_l(lo, hi, 11) & 0x7fffffffu;
    const unsigned long long m = ((unsigned long long)(mh | (e ? 0x80000000u : 0u)) << 32) | (lo << 11);
    unsigned long long v;
    asm("shr.u64 %0, %1, %2;" : "=l"(v) : "l"(m), "r"((uint32_t)(4 + E - max(e, 1))));  // 64 and more: 0
    v = (v + 1) >> 1;
    const long long sg = (long long)((int)hi >> 31);
    return (long long)((v ^ (unsigned long long)sg) - (unsigned long long)sg);
}
// v 2^e rounded to nearest, ties to even, v a number of a column under exponent
// E. tiny: a result can lie below the normal range (E < kTiny); e is then kUp
// more than it is, and a product by a power of two rounds once more.
constexpr int kTiny = 64, kUp = 128;
__device__ __forceinline__ double fix_out(long long v, int e, bool tiny) {
    const uint32_t sign = (uint32_t)(v >> 32) & 0x80000000u;
    const unsigned long long u = (unsigned long long)(v < 0 ? -v : v);
    const int lz = __clzll((long long)u);
    unsigned long long m = u << lz;
    m += 0x3ffull + ((m >> 11) & 1);
    const bool carry = m < 0x8000000000000000ull;
    const int be = 1023 + 63 - lz + e + (carry ? 1 : 0);
    if (u == 0) return 0.0;
    const unsigned long long f = carry ? 0 : ((m >> 11) & 0xfffffffffffffull);
    if (be >= 2047) return __hiloint2double((int)(sign | 0x7ff00000u), 0);
    const double r = __hiloint2double((int)(sign | ((uint32_t)be << 20) | (uint32_t)(f >> 32)), (int)(uint32_t)f);
    return tiny ? r * 2.938735877055719e-39 : r;  // 2^-kUp
}

__device__ __forceinline__ int fft_bexp(double2 v) {
    return (int)max(((uint32_t)__double2hiint(v.x) >> 20) & 0x7ffu, ((uint32_t)__double2hiint(v.y) >> 20) & 0x7ffu);
}

template <typename T> struct FftArith;
template <> struct FftArith<float> { typedef FftFloat type; };
template <> struct FftArith<double> { typedef FftFixed type; };

// ------------------------------------------------------------- transform
// One CTA: columns c = tid % bt (bt = 1 << lbt), items u = tid / bt. load(e)
// and store(k, v) as in fft_reg, by global type. S: shared [n][bt] of A::V,
// mx: shared int [bt] (double). Every thread of the block calls it.
template <typename T, int R, class Load>
__device__ __forceinline__ void gen_first(typename FftArith<T>::type::V *S, int *mx, const GenPlan &p, int lbt, int c,
                                          int u, bool swap, int &E, Load load) {
    typedef typename FftArith<T>::type A;
    C<T> raw[R];
    const int nr = p.n / R;
    const bool on = u < nr;
#pragma unroll
    for (int r = 0; r < R; r++) raw[r] = on ? load(u + r * nr) : mk<T>(0, 0);
    typename A::V v[R];
    if constexpr (sizeof(T) == sizeof(double)) {
        int e = 0;
#pragma unroll
        for (int r = 0; r < R; r++) e = max(e, fft_bexp(raw[r]));
        for (int o = 1 << lbt; o < 32; o <<= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
        if ((threadIdx.x & 31) < (1u << lbt)) atomicMax(&mx[c], e);
        __syncthreads();
        E = mx[c];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const long long a = fix_in(raw[r].x, E), b = fix_in(raw[r].y, E);
            v[r] = swap ? FixC{b, a} : FixC{a, b};
        }
    } else {
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = swap ? mk<T>(raw[r].y, raw[r].x) : raw[r];
    }
    Gdft<A, R>::run(v);
    if (on) {
#pragma unroll
        for (int r = 0; r < R; r++) S[((u * R + r) << lbt) + c] = v[r];
    }
    __syncthreads();
}

template <typename T, int R>
__device__ __forceinline__ void gen_read(typename FftArith<T>::type::V *v, const typename FftArith<T>::type::V *S,
                                         const GenPlan &p, int s, int lbt, int c, int j, int jm,
                                         const typename FftArith<T>::type::Tw *__restrict__ tw) {
    typedef typename FftArith<T>::type A;
    const int nr = p.n / R;
    const typename A::Tw *w = tw + p.off[s] + jm * (R - 1);
    v[0] = A::down(S[(j << lbt) + c], p.sh[s]);
#pragma unroll
    for (int r = 1; r < R; r++) v[r] = A::tw(S[((j + r * nr) << lbt) + c], w[r - 1], p.sh[s]);
    Gdft<A, R>::run(v);
}

template <typename T, int R>
__device__ __forceinline__ void gen_mid(typename FftArith<T>::type::V *S, const GenPlan &p, int s, int lbt, int c, int u,
                                        const typename FftArith<T>::type::Tw *__restrict__ tw) {
    const int Ns = p.Ns[s], jq = (int)(((uint32_t)u * (uint32_t)p.div[s]) >> 20), jm = u - jq * Ns;
    const bool on = u < p.n / R;
    typename FftArith<T>::type::V v[R];
    if (on) gen_read<T, R>(v, S, p, s, lbt, c, u, jm, tw);
    __syncthreads();
    if (on) {
#pragma unroll
        for (int r = 0; r < R; r++) S[((jq * Ns * R + jm + r * Ns) << lbt) + c] = v[r];
    }
    __syncthreads();
}

template <typename T, int R, class Store>
__device__ __forceinline__ void gen_last(const typename FftArith<T>::type::V *S, const GenPlan &p, int lbt, int c, int u,
                                         const typename FftArith<T>::type::Tw *__restrict__ tw, bool swap, int E,
                                         Store store) {
    const int s = p.ns - 1, nr = p.n / R;  // nr = Ns
    for (int j = u < p.rows ? u : nr; j < nr; j += p.rows) {
        typename FftArith<T>::type::V v[R];
        gen_read<T, R>(v, S, p, s, lbt, c, j, j, tw);
#pragma unroll
        for (int r = 0; r < R; r++) {
            if constexpr (sizeof(T) == sizeof(double)) {
                const bool bad = E == 2047, tiny = E < kTiny;
                const int e = E - 1081 + p.sh_sum + (tiny ? kUp : 0);
                const double a = bad ? (double)NAN : fix_out(v[r].x, e, tiny);
                const double b = bad ? (double)NAN : fix_out(v[r].y, e, tiny);
                store(j + r * nr, swap ? make_double2(b, a) : make_double2(a, b));
            } else {
                store(j + r * nr, swap ? mk<T>(v[r].y, v[r].x) : v[r]);
            }
        }
    }
}

// a stage of radix r, among the radices of the kernel's class: 0 {2, 4, 8},
// 1 {2..6, 8}, 2 {2..6, 8, 9, 10}, 3 {2..10} (registers go by the largest of
// the class)
#define EGX_RADIX(k, CALL) case k: { constexpr int R_ = k; CALL; break; }
#define EGX_RADIX_SWITCH(r, CALL)                                                                       \
    if constexpr (CLS == 0) {                                                                           \
        switch (r) { EGX_RADIX(2, CALL) EGX_RADIX(4, CALL) default: { constexpr int R_ = 8; CALL; } }    \
    } else if constexpr (CLS == 1) {                                                                    \
        switch (r) { EGX_RADIX(2, CALL) EGX_RADIX(3, CALL) EGX_RADIX(4, CALL) EGX_RADIX(5, CALL)        \
                     EGX_RADIX(6, CALL) default: { constexpr int R_ = 8; CALL; } }                      \
    } else if constexpr (CLS == 2) {                                                                    \
        switch (r) { EGX_RADIX(2, CALL) EGX_RADIX(3, CALL) EGX_RADIX(4, CALL) EGX_RADIX(5, CALL)        \
                     EGX_RADIX(6, CALL) EGX_RADIX(8, CALL) EGX_RADIX(9, CALL)                           \
                     default: { constexpr int R_ = 10; CALL; } }                                        \
    } else {                                                                                            \
        switch (r) { EGX_RADIX(2, CALL) EGX_RADIX(3, CALL) EGX_RADIX(4, CALL) EGX_RADIX(5, CALL)        \
                     EGX_RADIX(6, CALL) EGX_RADIX(7, CALL) EGX_RADIX(8, CALL) EGX_RADIX(9, CALL)        \
                     default: { constexpr int R_ = 10; CALL; } }                                        \
    }

template <typename T, int CLS, class Load, class Store>
__device__ __forceinline__ void fft_gen(unsigned char *smem, const GenPlan &p, int lbt,
                                        const C<T> *__restrict__ table, int sign, Load load, Store store) {
    typedef typename FftArith<T>::type A;
    typename A::V *S = reinterpret_cast<typename A::V *>(smem);
    int *mx = reinterpret_cast<int *>(smem + ((size_t)p.n << lbt) * sizeof(typename A::V));
    const typename A::Tw *tw = reinterpret_cast<const typename A::Tw *>(table + p.n);
    const int c = threadIdx.x & ((1 << lbt) - 1), u = threadIdx.x >> lbt;
    const bool swap = sign > 0;
    int E = 0;
    if (sizeof(T) == sizeof(double)) {
        if (threadIdx.x < (1u << lbt)) mx[threadIdx.x] = 0;
        __syncthreads();
    }
    EGX_RADIX_SWITCH(p.R[0], (gen_first<T, R_>(S, mx, p, lbt, c, u, swap, E, load)))
    for (int s = 1; s + 1 < p.ns; s++) {
        EGX_RADIX_SWITCH(p.R[s], (gen_mid<T, R_>(S, p, s, lbt, c, u, tw)))
    }
    EGX_RADIX_SWITCH(p.R[p.ns - 1], (gen_last<T, R_>(S, p, lbt, c, u, tw, swap, E, store)))
}

// block size and resident blocks the kernels are compiled for: 64 registers
// (complex128) and 32; the large radices spill some of theirs, and four
// blocks still hide more latency than three or two without (240-point
// complex128 lines 152 against 172 and 209 us, 360-point complex64 lines 76
// against 82 and 97)
template <typename T, int CLS> constexpr int gen_max_threads() { return sizeof(T) == sizeof(double) ? 256 : 512; }
template <typename T, int CLS> constexpr int gen_min_blocks() { return 4; }

// Host: log2 of the columns per CTA, the block and its shared memory.
struct GenLaunch {
    int lbt, threads;
    size_t smem;
};
template <typename T> inline GenLaunch gen_launch(const GenPlan &p, int lbt) {
    GenLaunch l;
    l.lbt = lbt;
    l.threads = ((p.rows << l.lbt) + 31) / 32 * 32;
    l.smem = ((size_t)p.n << l.lbt) * sizeof(C<T>) + (16 << 2);
    return l;
}
// complex128: 4 columns (64-byte rows), complex64 8, fewer where the block's
// threads or an idle GPU ask for it
template <typename T> inline GenLaunch gen_launch(const GenPlan &p, int B, int nlines) {
    int lbt = sizeof(T) == sizeof(double) ? 2 : 3;
    while (lbt > 0 && (p.rows << lbt) > gen_max_threads<T, 0>()) lbt--;
    while (lbt > 1 && (long)((B + (1 << lbt) - 1) >> lbt) * nlines < 4 * 152) lbt--;
    return gen_launch<T>(p, lbt);
}

}  // namespace egx
