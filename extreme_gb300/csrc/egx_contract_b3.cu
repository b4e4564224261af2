// complex64 block contraction of the CIE operator
// (ConvolutionOperator.ApplyGreenTensorAlongZ, ConvolutionOperator.cs:274-327)
// for the packed Green layout (layer counts without the sub-block layout, up
// to 48) on the BF16 tensor cores.
//
// Every operand is the sum of three BF16 parts, h + m + l: 24 bits, an FP32
// value exactly, and over the whole FP32 range, since BF16 has its exponent
// (Henry, Tang and Heinecke, "Leveraging the bfloat16 artificial intelligence
// datatype for higher-precision computations", ARITH 2019). The products h h,
// h m, m h, m m, h l and l h are kept; the others lie below 2^-25 of their
// term. So an entry keeps its bits however small it is beside the others of
// its row, column or vector (a source in one layer, a tensor that falls
// exponentially with the distance of two layers). The tensor cores' FP32
// accumulators truncate: the products h h of 16 columns are added to the sum
// by rounded additions, and the small products have accumulators of their own.
//
// Algebra as in egx_contract.cu: the (up to) four spectral points that share a
// stored block are right-hand sides of one matrix after the D_p sign flips; its
// z rows hold -A^T where its z columns hold A. The eight columns of an MMA are
// the real and imaginary parts of the four points, Gr [Xr | Xi] and
// Gi [Xr | Xi], side by side in a lane, which joins and stores them.
//
// One CTA per stored point (grid-stride), a warp per 16-row tile. The block
// comes by one bulk copy; a lane's entries of a tile are loaded from the places
// in a table (egx_diglayout.cuh) and split in registers, once for the two
// right-hand sides of a pass.
//
// Measured at 180x120x35, two right-hand sides: 549 us per launch (2.1 TB/s of
// tensor and buffer), one 400; the FP32 kernel (k_contract_c64) 1,647 and 977.
// 90x75x22, two: 88 us against 338. Bound by latency: the table and the
// fragments leave room for 14 warps per SM at 35 layers, which fill 48 % of the
// issue slots (tensor pipe 31 %, DRAM 24 %, 64x64x35). 2-norm error of an apply
// against 64 bits, 64x60 cells, 4..47 layers: 2.9e-8..4.4e-8 where the FP32
// kernels' is 2.9e-8..6.5e-8.
#include <cuda_bf16.h>

#include <algorithm>
#include <cstdint>

#include "egx_diglayout.cuh"
#include "egx_operator.cuh"
#include "egx_wait.cuh"

namespace egx {

namespace {

constexpr uint64_t kWait = 2000000000ull;

__device__ __forceinline__ void mma_bf16(float *c, const uint32_t *a, uint2 b) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y));
}

// the next part of (a, b) as a pair, taken off them
__device__ __forceinline__ uint32_t take_part(float &a, float &b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    const uint32_t w = *reinterpret_cast<const uint32_t *>(&h);
    a -= __uint_as_float(w << 16);
    b -= __uint_as_float(w & 0xffff0000u);
    return w;
}

// shared memory: block, fragments [KT][NR][3 parts][32 lanes], places
struct Geom {
    int np, MT;
    uint32_t point, o_tab, bytes;
};
__host__ __device__ inline Geom geom(int nz, int NR) {
    Geom g;
    g.np = (nz + 1) & ~1;
    g.MT = (3 * g.np + 15) / 16;
    g.point = (uint32_t)(4 * nz * (nz + 1)) * 8u;
    g.o_tab = g.point + (uint32_t)(g.MT * NR * 3) * 256u;
    g.bytes = g.o_tab + (uint32_t)(g.MT * g.MT) * 512u;
    return g;
}

template <int NR, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB)
    k_contract_b3(float2 *buf, const float2 *__restrict__ G, const OpDims d, int *err) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t bar;
    const Geom m = geom(d.nz, NR);
    const int nz = d.nz, R = 3 * nz, MT = m.MT, KT = m.MT;
    uint2 *bfr = reinterpret_cast<uint2 *>(smem + m.point);
    uint4 *tab = reinterpret_cast<uint4 *>(smem + m.o_tab);
    const int tid = threadIdx.x, lane = tid & 31, mt = tid >> 5, g = lane >> 2, t = lane & 3;
    const int Q = (d.nx + 1) * (d.ny + 1), n1 = 2 * d.ny;
    const uint32_t sbar = (uint32_t)__cvta_generic_to_shared(&bar), sG = (uint32_t)__cvta_generic_to_shared(smem);

    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sbar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // a lane's entries of a tile: rows g and g + 8, columns 2t, 2t + 1 and 8
    // on; the flag where the matrix has the entry's negative (z rows of xz, yz)
    for (int i = tid; i < MT * KT * 32; i += blockDim.x) {
        const int ln = i & 31, tile = i >> 5, tm = tile / KT, r = 16 * tm + (ln >> 2);
        const int c = 16 * (tile - tm * KT) + 2 * (ln & 3);
        auto word = [&](int row, int col) {
            const uint32_t w = dig_word(nz, row, col);
            return row / m.np == 2 ? w : w & ~0x8000u;
        };
        tab[i] = make_uint4(word(r, c), word(r + 8, c), word(r, c + 8), word(r + 8, c + 8));
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

    // this thread's right-hand-side entries: point xv, rows xj and xj + 8 MT
    const int xv = tid & 3, xmx = xv >> 1, xmy = xv & 1;
    auto load_x = [&](int q, int rhs, int j) {
        const int c = j / m.np, k = j - c * m.np;
        const int a = q / (d.ny + 1), bq = q - a * (d.ny + 1);
        const int nkx = (a == 0 || a == d.nx) ? 1 : 2;
        const int nky = (bq == 0 || bq == d.ny) ? 1 : 2;
        if (c > 2 || k >= nz || xmx >= nkx || xmy >= nky || rhs >= d.nrhs) return make_float2(0.f, 0.f);
        const long pt = (long)(xmx ? 2 * d.nx - a : a) * n1 + (xmy ? 2 * d.ny - bq : bq);
        const float2 x = buf[pt * d.B + rhs * R + c * nz + k];
        return (c == 0 && xmx) || (c == 1 && xmy) ? make_float2(-x.x, -x.y) : x;
    };
    float2 xnext[NR][2];
    auto load_next = [&](int q, int rhs) {
#pragma unroll
        for (int r = 0; r < NR; r++)
#pragma unroll
            for (int h = 0; h < 2; h++) xnext[r][h] = load_x(q, rhs + r, (tid >> 2) + h * 8 * MT);
    };
    if ((int)blockIdx.x < Q) load_next(blockIdx.x, 0);
    uint32_t phase = 0;
    for (int q = blockIdx.x; q < Q; q += gridDim.x) {
        const int a = q / (d.ny + 1), bq = q - a * (d.ny + 1);
        const int nkx = (a == 0 || a == d.nx) ? 1 : 2;
        const int nky = (bq == 0 || bq == d.ny) ? 1 : 2;
        for (int rhs = 0; rhs < d.nrhs; rhs += NR) {
#pragma unroll
            for (int r = 0; r < NR; r++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    // columns 2 xv (real) and 2 xv + 1, row j of a part's fragment
                    const int j = (tid >> 2) + h * 8 * MT;
                    uint16_t *o = reinterpret_cast<uint16_t *>(bfr) + ((j >> 4) * NR + r) * (3 * 128) +
                                  (8 * xv + ((j & 7) >> 1)) * 4 + ((j >> 3) & 1) * 2 + (j & 1);
                    float2 x = xnext[r][h];
#pragma unroll
                    for (int p = 0; p < 3; p++) {
                        const uint32_t w = take_part(x.x, x.y);
                        o[p * 128] = (uint16_t)w;
                        o[p * 128 + 16] = (uint16_t)(w >> 16);
                    }
                }
            if (rhs == 0) {
                const bool late = !mbar_wait_ns(sbar, phase, kWait);
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
            // the next pass's loads, and the next point's block on its way into
            // L2, while this one is multiplied
            if (rhs + NR < d.nrhs) {
                load_next(q, rhs + NR);
            } else if (q + (int)gridDim.x < Q) {
                load_next(q + gridDim.x, 0);
                if (tid == 0)
                    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(
                                     reinterpret_cast<const unsigned char *>(G) + (size_t)(q + gridDim.x) * m.point),
                                 "r"(m.point)
                                 : "memory");
            }

            float big[NR][2][4] = {}, low[NR][2][4] = {};  // Gr X, Gi X: h h, the small products
            const uint2 *bp = bfr + lane;
            const float2 *M = reinterpret_cast<const float2 *>(smem);
#pragma unroll 1
            for (int kt = 0; kt < KT; kt++) {
                const uint4 w = tab[(mt * KT + kt) * 32 + lane];
                uint32_t ap[2][3][4];  // plane, part
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const uint32_t wk = k == 0 ? w.x : k == 1 ? w.y : k == 2 ? w.z : w.w;
                    const uint32_t flip = (wk & 0x8000u) << 16;
                    const float2 u = M[wk & 0x3fffu], v = M[wk >> 16];
                    auto sg = [&](float f) { return __uint_as_float(__float_as_uint(f) ^ flip); };
                    float ur = sg(u.x), ui = sg(u.y), vr = sg(v.x), vi = sg(v.y);
#pragma unroll
                    for (int p = 0; p < 3; p++) ap[0][p][k] = take_part(ur, vr), ap[1][p][k] = take_part(ui, vi);
                }
#pragma unroll
                for (int r = 0; r < NR; r++) {
                    uint2 b[3];
#pragma unroll
                    for (int p = 0; p < 3; p++) b[p] = bp[((kt * NR + r) * 3 + p) * 32];
#pragma unroll
                    for (int c = 0; c < 2; c++) {
                        float s[4] = {};
                        mma_bf16(s, ap[c][0], b[0]);
                        mma_bf16(low[r][c], ap[c][2], b[0]);
                        mma_bf16(low[r][c], ap[c][1], b[1]);
                        mma_bf16(low[r][c], ap[c][0], b[2]);
                        mma_bf16(low[r][c], ap[c][1], b[0]);
                        mma_bf16(low[r][c], ap[c][0], b[1]);
#pragma unroll
                        for (int i = 0; i < 4; i++) big[r][c][i] += s[i];
                    }
                }
            }
            __syncthreads();  // the fragments and the block are read
            if (tid == 0 && rhs + NR >= d.nrhs && q + (int)gridDim.x < Q) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                fetch(q + gridDim.x);
            }
            // this lane's rows g, g + 8 of point t
            const int ymx = t >> 1, ymy = t & 1;
            if (ymx < nkx && ymy < nky) {
                const long pt = (long)(ymx ? 2 * d.nx - a : a) * n1 + (ymy ? 2 * d.ny - bq : bq);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int row = 16 * mt + g + 8 * h, rc = row / m.np, rk = row - rc * m.np;
                    if (rc > 2 || rk >= nz) continue;
                    const bool flip = (rc == 0 && ymx) || (rc == 1 && ymy);
#pragma unroll
                    for (int r = 0; r < NR; r++) {
                        if (NR > 1 && rhs + r >= d.nrhs) continue;
                        const float *p = big[r][0] + 2 * h, *s = big[r][1] + 2 * h;
                        const float *pl = low[r][0] + 2 * h, *sl = low[r][1] + 2 * h;
                        float2 y = make_float2((p[0] - s[1]) + (pl[0] - sl[1]), (p[1] + s[0]) + (pl[1] + sl[0]));
                        if (flip) y = make_float2(-y.x, -y.y);
                        buf[pt * d.B + (rhs + r) * R + rc * nz + rk] = y;
                    }
                }
            }
        }
    }
}

template <int NR, int MAXT, int MINB>
void launch(float2 *buf, const float2 *G, const OpDims &d, int *err, cudaStream_t s) {
    static const int nsm = [] {
        int n = 0;
        EGX_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, 0));
        return n;
    }();
    const Geom m = geom(d.nz, NR);
    const auto kernel = k_contract_b3<NR, MAXT, MINB>;
    raise_smem_limit((const void *)kernel, m.bytes);
    const int thr = 32 * m.MT;
    int per = 0;
    EGX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, thr, m.bytes));
    const long Q = (long)(d.nx + 1) * (d.ny + 1);
    const unsigned grid = (unsigned)std::min<long>(Q, (long)nsm * std::max(1, per));
    launch_after(buffer_bytes<float>(d), kernel, grid, thr, m.bytes, s, buf, G, d, err);
}

}  // namespace

bool contract_b3_fits(int nz) { return nz <= 48; }

void launch_contract_b3(float2 *buf, const float2 *G, const OpDims &d, int *err, cudaStream_t s) {
    if (d.nrhs == 1) launch<1, 288, 2>(buf, G, d, err, s);
    else launch<2, 288, 2>(buf, G, d, err, s);
}

}  // namespace egx
