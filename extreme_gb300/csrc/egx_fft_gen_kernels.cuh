// Kernels of the generic transform (egx_fft_gen.cuh): the operator's y passes
// with their factors, plain lines, and lines stored by half under a parity;
// and their launches, instantiated for complex64 in egx_fft_gen32.cu and for
// complex128 in egx_fft_gen64.cu.
#pragma once

#include <type_traits>

#include "egx_fft_gen.cuh"
#include "egx_operator.cuh"

namespace egx {

namespace {

// rx = r x scaled by the forward factors (real), zero-padded, DFT along y
template <typename T, int CLS>
__global__ void __launch_bounds__(gen_max_threads<T, CLS>(), gen_min_blocks<T, CLS>())
    k_fwd_y_g(const C<T> *__restrict__ x, const OperatorData<T> op, C<T> *__restrict__ buf, const OpDims d,
              const GenPlan p, const C<T> *__restrict__ tw, int lbt) {
    extern __shared__ __align__(16) unsigned char smem[];
    after_previous();
    const int i = blockIdx.y, b = (blockIdx.x << lbt) + (threadIdx.x & ((1 << lbt) - 1));
    const bool bok = b < d.B;
    const int per = 3 * d.nz;
    const int rhs = bok ? b / per : 0, rem = b - rhs * per, k = rem % d.nz;
    const T f = bok ? op.fwd[k].x : T(0);
    const C<T> *xr = x + rhs * d.nvec + (long)i * d.ny * per + rem;
    const C<T> *rr = op.r + (long)i * d.ny * d.nz + k;
    auto load = [&](int j) -> C<T> {
        if (!bok || j >= d.ny) return mk<T>(0, 0);
        return cscale<T>(cmul<T>(rr[(long)j * d.nz], xr[(long)j * per]), f);
    };
    C<T> *row = buf + (long)i * p.n * d.B + b;
    auto store = [&](int j, C<T> v) {
        if (bok) row[(long)j * d.B] = v;
    };
    fft_gen<T, CLS>(smem, p, lbt, tw, -1, load, store);
}

template <typename T, int CLS>
__global__ void __launch_bounds__(gen_max_threads<T, CLS>(), gen_min_blocks<T, CLS>())
    k_lines_g(C<T> *buf, long lstride, long estride, int B, int nload, int nstore, const GenPlan p,
              const C<T> *__restrict__ tw, int lbt, int sign) {
    extern __shared__ __align__(16) unsigned char smem[];
    after_previous();
    const int b = (blockIdx.x << lbt) + (threadIdx.x & ((1 << lbt) - 1));
    const bool bok = b < B;
    C<T> *line = buf + (long)blockIdx.y * lstride + b;
    auto load = [&](int e) -> C<T> { return (bok && e < nload) ? line[e * estride] : mk<T>(0, 0); };
    auto store = [&](int e, C<T> v) {
        if (bok && e < nstore) line[e * estride] = v;
    };
    fft_gen<T, CLS>(smem, p, lbt, tw, sign, load, store);
}

// inverse DFT along y, backward factors (real) and the last step
template <typename T, int CLS>
__global__ void __launch_bounds__(gen_max_threads<T, CLS>(), gen_min_blocks<T, CLS>())
    k_bwd_y_g(const C<T> *__restrict__ buf, const C<T> *__restrict__ x, const OperatorData<T> op,
              C<T> *__restrict__ y, const OpDims d, const GenPlan p, const C<T> *__restrict__ tw, int lbt) {
    extern __shared__ __align__(16) unsigned char smem[];
    after_previous();
    const int i = blockIdx.y, b = (blockIdx.x << lbt) + (threadIdx.x & ((1 << lbt) - 1));
    const bool bok = b < d.B;
    const int per = 3 * d.nz;
    const int rhs = bok ? b / per : 0, rem = b - rhs * per, k = rem % d.nz;
    const T bw = bok ? op.bwd[k].x : T(0);
    const C<T> *row = buf + (long)i * p.n * d.B + b;
    auto load = [&](int j) -> C<T> { return bok ? row[(long)j * d.B] : mk<T>(0, 0); };
    auto store = [&](int j, C<T> v) {
        if (!bok || j >= d.ny) return;
        const long cell = (long)i * d.ny + j;
        const long idx = rhs * d.nvec + cell * per + rem;
        const C<T> yv = cscale<T>(v, bw);
        const C<T> xv = x[idx];
        const C<T> rx = cmul<T>(op.r[cell * d.nz + k], xv);
        y[idx] = (op.type == EGX_OP_A) ? csub<T>(csub<T>(xv, yv), rx) : cadd<T>(yv, rx);
    };
    fft_gen<T, CLS>(smem, p, lbt, tw, +1, load, store);
}

dim3 gen_grid(int B, int lbt, int nlines) { return dim3((B + (1 << lbt) - 1) >> lbt, nlines); }

template <class Run> void by_class(const GenPlan &p, Run run) {
    if (p.cls == 0) run(std::integral_constant<int, 0>{});
    else if (p.cls == 1) run(std::integral_constant<int, 1>{});
    else if (p.cls == 2) run(std::integral_constant<int, 2>{});
    else run(std::integral_constant<int, 3>{});
}

bool gen_ok(const GenPlan &p, int nlines) { return p.ns > 0 && nlines <= 65535; }

}  // namespace

template <typename T>
bool gen_fwd_y(const FftPlan &p, const C<T> *x, const OperatorData<T> &op, C<T> *buf, const OpDims &d, const C<T> *tw,
               cudaStream_t s) {
    if (!gen_ok(p.gen, d.nx)) return false;
    const GenLaunch l = gen_launch<T>(p.gen, d.B, d.nx);
    auto run = [&](auto cls) {
        constexpr int K = decltype(cls)::value;
        raise_smem_limit((const void *)k_fwd_y_g<T, K>, l.smem);
        launch_after(buffer_bytes<T>(d), k_fwd_y_g<T, K>, gen_grid(d.B, l.lbt, d.nx), l.threads, l.smem, s, x, op, buf,
                     d, p.gen, tw, l.lbt);
    };
    by_class(p.gen, run);
    return true;
}

template <typename T>
bool gen_bwd_y(const FftPlan &p, const C<T> *buf, const C<T> *x, const OperatorData<T> &op, C<T> *y, const OpDims &d,
               const C<T> *tw, cudaStream_t s) {
    if (!gen_ok(p.gen, d.nx)) return false;
    const GenLaunch l = gen_launch<T>(p.gen, d.B, d.nx);
    auto run = [&](auto cls) {
        constexpr int K = decltype(cls)::value;
        raise_smem_limit((const void *)k_bwd_y_g<T, K>, l.smem);
        launch_after(buffer_bytes<T>(d), k_bwd_y_g<T, K>, gen_grid(d.B, l.lbt, d.nx), l.threads, l.smem, s, buf, x, op,
                     y, d, p.gen, tw, l.lbt);
    };
    by_class(p.gen, run);
    return true;
}

template <typename T>
bool gen_lines(const FftPlan &p, C<T> *buf, int nlines, long lstride, long estride, int B, int nload, int nstore,
               const C<T> *tw, int sign, cudaStream_t s) {
    if (!gen_ok(p.gen, nlines)) return false;
    const GenLaunch l = gen_launch<T>(p.gen, B, nlines);
    auto run = [&](auto cls) {
        constexpr int K = decltype(cls)::value;
        raise_smem_limit((const void *)k_lines_g<T, K>, l.smem);
        launch_after((size_t)nlines * p.n * B * sizeof(C<T>), k_lines_g<T, K>, gen_grid(B, l.lbt, nlines), l.threads,
                     l.smem, s, buf, lstride, estride, B, nload, nstore, p.gen, tw, l.lbt, sign);
    };
    by_class(p.gen, run);
    return true;
}

#define EGX_GEN_INST(T)                                                                                              \
    template bool gen_fwd_y<T>(const FftPlan &, const C<T> *, const OperatorData<T> &, C<T> *, const OpDims &,       \
                               const C<T> *, cudaStream_t);                                                          \
    template bool gen_bwd_y<T>(const FftPlan &, const C<T> *, const C<T> *, const OperatorData<T> &, C<T> *,         \
                               const OpDims &, const C<T> *, cudaStream_t);                                          \
    template bool gen_lines<T>(const FftPlan &, C<T> *, int, long, long, int, int, int, const C<T> *, int, cudaStream_t);

}  // namespace egx
