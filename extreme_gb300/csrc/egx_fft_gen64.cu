// The generic transform's complex128 kernels and its twiddle tables.
#include <cmath>

#include "egx_fft_gen_kernels.cuh"

namespace egx {

namespace {

// lines whose second half is the parity image of the first (see k_lines_sym_r)
template <int CLS>
__global__ void __launch_bounds__(gen_max_threads<double, CLS>(), gen_min_blocks<double, CLS>())
    k_lines_sym_g(double2 *buf, long lstride, long estride, int B, int parity, int nstore, const GenPlan p,
                  const double2 *__restrict__ tw, int lbt, int sign) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int b = (blockIdx.x << lbt) + (threadIdx.x & ((1 << lbt) - 1));
    const bool bok = b < B;
    const int NH = p.n / 2;
    double2 *line = buf + (long)blockIdx.y * lstride + b;
    auto load = [&](int e) -> double2 {
        if (!bok || e == NH) return make_double2(0, 0);
        const double2 v = line[(e < NH ? e : p.n - e) * estride];
        return e > NH && parity < 0 ? make_double2(-v.x, -v.y) : v;
    };
    auto store = [&](int e, double2 v) {
        if (bok && e < nstore) line[e * estride] = v;
    };
    fft_gen<double, CLS>(smem, p, lbt, tw, sign, load, store);
}

}  // namespace

bool gen_lines_sym(const FftPlan &p, double2 *buf, int nlines, long lstride, long estride, int B, int parity,
                   int nstore, const double2 *tw, int sign, cudaStream_t s) {
    if (!gen_ok(p.gen, nlines)) return false;
    const GenLaunch l = gen_launch<double>(p.gen, B, nlines);
    auto run = [&](auto cls) {
        constexpr int K = decltype(cls)::value;
        raise_smem_limit((const void *)k_lines_sym_g<K>, l.smem);
        k_lines_sym_g<K><<<gen_grid(B, l.lbt, nlines), l.threads, l.smem, s>>>(buf, lstride, estride, B, parity,
                                                                                nstore, p.gen, tw, l.lbt, sign);
    };
    by_class(p.gen, run);
    return true;
}

namespace {

// exp(-2 pi i k / n) for k < n, each angle reduced to the nearest quarter turn
// (|angle| <= 1/8 turn, evaluated once per size)
struct Roots {
    std::vector<long double> c, s;
    explicit Roots(int n) : c(n), s(n) {
        const long double tau = 6.283185307179586476925286766559005768L;
        std::vector<long double> ca(n / 2 + 1, 2.0L), sa(n / 2 + 1);
        for (int k = 0; k < n; k++) {
            const long o = (8L * k / n + 1) / 2, r = 4L * k - o * n, ar = r < 0 ? -r : r;
            if (ca[ar] > 1.5L) {
                const long double a = tau * (long double)ar / (4.0L * n);
                ca[ar] = cosl(a);
                sa[ar] = sinl(a);
            }
            const long double x = ca[ar], y = r < 0 ? -sa[ar] : sa[ar];
            // e^{i (a + q pi / 2)}, conjugated
            const int q = (int)(o & 3);
            c[k] = q == 0 ? x : (q == 1 ? -y : (q == 2 ? -x : y));
            s[k] = -(q == 0 ? y : (q == 1 ? x : (q == 2 ? -y : -x)));
        }
    }
};

// f(entry, root, shift) over the stage table of a plan; the twiddles of every
// stage are n-th roots
template <class F> void stage_table(const GenPlan &p, F f) {
    for (int s = 1; s < p.ns; s++)
        for (int jm = 0; jm < p.Ns[s]; jm++)
            for (int r = 1; r < p.R[s]; r++)
                f((size_t)p.off[s] + jm * (p.R[s] - 1) + r - 1, jm * r * (p.n / (p.Ns[s] * p.R[s])), p.sh[s]);
}

}  // namespace

std::vector<double> fft_table64(int n) {
    std::vector<double> t = twiddles(n);
    const GenPlan p = make_gen_plan(n);
    t.resize(4 * (size_t)n, 0.0);
    if (!p.ns) return t;
    const Roots w(n);
    int *o = reinterpret_cast<int *>(t.data() + 2 * (size_t)n);
    auto put = [](long double v, int sh, int *x) {
        const long double f = ldexpl(v, 32 - sh), h = roundl(f), l = roundl(ldexpl(f - h, 32));
        x[0] = (int)h;
        x[1] = (int)(l > 2147483647.0L ? 2147483647.0L : (l < -2147483647.0L ? -2147483647.0L : l));
    };
    stage_table(p, [&](size_t e, int k, int sh) {
        put(w.c[k], sh, o + 4 * e);
        put(w.s[k], sh, o + 4 * e + 2);
    });
    return t;
}

std::vector<float> fft_table32(int n) {
    const std::vector<double> t = twiddles(n);
    std::vector<float> f(t.begin(), t.end());
    f.resize(4 * (size_t)n, 0.f);
    stage_table(make_gen_plan(n), [&](size_t e, int k, int) {
        f[2 * ((size_t)n + e)] = (float)t[2 * (size_t)k];
        f[2 * ((size_t)n + e) + 1] = (float)t[2 * (size_t)k + 1];
    });
    return f;
}

EGX_GEN_INST(double)

}  // namespace egx
