// Layer kernels of the learned preconditioner's network (egx_learn.cu): the
// passes over whole activations, (samples x depth x lateral cells) rows of W
// FP32 channels, 537 MB each at 8 samples of 128x128x32 and W = 32. They do a
// few operations per byte, so each is written to read every activation once,
// in 16-byte loads that go straight from memory into the operand registers of
// mma.sync m16n8k16 (BF16 operands, FP32 accumulators): the order of the
// contracted index and of the columns within a tile is free, so a lane takes
// the four (or eight) consecutive floats that it loads as its share of a
// fragment, and no tile is staged in shared memory.
//
// Two lane layouts of a 16-deep step, lane = 4 g + t:
//   rows    contracted index = memory row: rows 4t .. 4t + 3, columns
//           4g .. 4g + 3 of 32 (column 4g + j is column g of n-tile j)
//   cols    contracted index = memory column: columns 4t .. 4t + 3 of 16
// With either, the accumulators of the four n-tiles hold columns 8t .. 8t + 7
// of a row: two 16-byte stores.
//
// Measured at 8 samples of 128x128x32, W = 32, per layer (before: the strided
// GEMM with element loads, k_gemm_bf16, and separate element-wise passes):
//   lateral analysis   98 us (5.5 TB/s)                       before 391
//   layer sums         434 us forward (3.7 TB/s with the sums
//                      before the activation kept), 340 us
//                      backward (two blocks per SM; three spill:
//                      567, 460)                              3,200 and 2,167
//   weight gradient    458 us with gelu' and the column sums,
//                      236 us without (4.6 TB/s)              6,076 and 5,775
//   depth gradient     158 us (6.8 TB/s)                      3,320
#include <cuda_bf16.h>

#include <algorithm>
#include <cstdint>

#include "egx_common.cuh"
#include "egx_learn.cuh"

namespace egx {

namespace {

constexpr int KM = kNetModes;

__device__ __forceinline__ uint32_t pack(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}

__device__ __forceinline__ void mma(float *c, const uint32_t *a, const uint32_t *b) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ float comp(const float4 &v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
__device__ __forceinline__ float4 ld4(const float *p, bool on) {
    return on ? *reinterpret_cast<const float4 *>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
}

// the B fragments of four n-tiles from four rows (layout `rows`)
__device__ __forceinline__ void b_rows(uint32_t (*b)[2], const float4 *v) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
        b[j][0] = pack(comp(v[0], j), comp(v[1], j));
        b[j][1] = pack(comp(v[2], j), comp(v[3], j));
    }
}

// accumulators of a row's columns 8t .. 8t + 7 (h = 0: row g, 1: row g + 8)
__device__ __forceinline__ float4 acc_lo(const float (*c)[4], int h) {
    return make_float4(c[0][2 * h], c[1][2 * h], c[2][2 * h], c[3][2 * h]);
}
__device__ __forceinline__ float4 acc_hi(const float (*c)[4], int h) {
    return make_float4(c[0][2 * h + 1], c[1][2 * h + 1], c[2][2 * h + 1], c[3][2 * h + 1]);
}

// fragments of a 16 x (16 steps) A operand, rows m0.. of `rows`, `K` deep:
// word 32 (step) + lane, contracted index 16 step + 4t + i in slot i
template <typename F>
__device__ __forceinline__ void a_fragments(uint4 *dst, int steps, int tid, int threads, F at) {
    for (int e = tid; e < steps * 32; e += threads) {
        const int s = e >> 5, g = (e & 31) >> 2, k = 16 * s + 4 * (e & 3);
        dst[e] = make_uint4(pack(at(g, k), at(g, k + 1)), pack(at(g + 8, k), at(g + 8, k + 1)),
                            pack(at(g, k + 2), at(g, k + 3)), pack(at(g + 8, k + 2), at(g + 8, k + 3)));
    }
}

// ------------------------------------------------------- lateral analysis
// out[b][i][n] = sum_k bas[k][i] in[b][k][n], i < 16: the basis's columns
// against K rows of N contiguous columns (rows ks apart). A warp per batch
// item and 32 columns; the basis lies in shared memory as A fragments.
__global__ void __launch_bounds__(256, 3) k_analysis(const float *__restrict__ bas, const float *__restrict__ in, int K,
                                                  long ks, long in_b, int N, long items, float *__restrict__ out) {
    extern __shared__ uint4 fr[];
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, steps = (K + 15) / 16;
    a_fragments(fr, steps, threadIdx.x, 256, [&](int i, int k) { return k < K ? bas[(long)k * KM + i] : 0.f; });
    __syncthreads();
    const int chunks = (N + 31) / 32;
    for (long it = (long)blockIdx.x * 8 + (threadIdx.x >> 5); it < items; it += (long)gridDim.x * 8) {
        const long b = it / chunks;
        const int n0 = (int)(it - b * chunks) * 32;
        const bool in_n = n0 + 4 * g < N;
        const float *p = in + b * in_b + n0 + 4 * g + 4 * t * ks;
        float acc[4][4] = {};
#pragma unroll 4
        for (int s = 0; s < steps; s++, p += 16 * ks) {
            float4 v[4];
#pragma unroll
            for (int j = 0; j < 4; j++) v[j] = ld4(p + j * ks, in_n && 16 * s + 4 * t + j < K);
            uint32_t bf[4][2];
            b_rows(bf, v);
            const uint4 a4 = fr[s * 32 + lane];
            const uint32_t a[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
            for (int j = 0; j < 4; j++) mma(acc[j], a, bf[j]);
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            float *o = out + (b * KM + g + 8 * h) * N + n0 + 8 * t;
            if (n0 + 8 * t < N) *reinterpret_cast<float4 *>(o) = acc_lo(acc, h);
            if (n0 + 8 * t + 4 < N) *reinterpret_cast<float4 *>(o + 4) = acc_hi(acc, h);
        }
    }
}

// ------------------------------------------------------------- layer sums
// The three branches of a layer in one pass over its input (and, with
// transposed weights, of its gradient):
//   out[z, cell, c] = sum_z' D(z, z') in[z', cell, c] + sum_k in[z, cell, k] Wt(k, c)
//                   + sum_j bas[i, j] sp[z, outer, j, c]   (+ bias[c]), cell = (outer, i)
// A block takes 16 cells along the basis's direction and 32 channels; its
// eight warps first write the lateral branch of up to 32 depths into shared
// memory (the basis against 16 modes, one MMA row tile per depth), then take
// two cells each: the cell's depths x channels block is the `rows` operand of
// the depth mixing and the `cols` operand of the channel mixing. Each branch
// is summed by itself and they are joined in the order of the separate
// products (lateral + channel, + depth, + bias): the general path's sums to
// the bit, so that no BF16 operand of a later layer rounds the other way.
struct LayerK {
    NetLayer a;
    int tiles_line, zc;   // 16-cell tiles per line; 32-depth chunks
    uint32_t o_d, o_w;    // shared memory: D's and Wt's fragments, in bytes
    long tiles;
};

constexpr uint32_t kSpecBytes = 32 * 16 * 32 * 4;

template <bool PRE, bool ACT>
__global__ void __launch_bounds__(256, 2) k_layer(const LayerK q) {
    extern __shared__ __align__(16) unsigned char sm[];
    const NetLayer &a = q.a;
    float4 *spec = reinterpret_cast<float4 *>(sm);
    uint4 *df = reinterpret_cast<uint4 *>(sm + q.o_d);
    uint2 *wf = reinterpret_cast<uint2 *>(sm + q.o_w);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int nz = a.nz, W = a.W, c0 = blockIdx.y * 32, zs = (nz + 15) / 16, ws = (W + 15) / 16;
    const long slab = a.ncell * W;
    for (int m = 0; m < 2 * q.zc; m++)
        a_fragments(df + m * zs * 32, zs, tid, 256, [&](int i, int k) {
            return 16 * m + i < nz && k < nz ? a.D[(16 * m + i) * a.d_o + k * a.d_i] : 0.f;
        });
    for (int e = tid; e < ws * 4 * 32; e += 256) {
        const int s = e >> 7, c = c0 + 4 * ((e & 31) >> 2) + ((e >> 5) & 3), k = 16 * s + 4 * (e & 3);
        float w[4];
#pragma unroll
        for (int i = 0; i < 4; i++) w[i] = c < W && k + i < W ? a.Wt[(k + i) * a.w_k + c * a.w_n] : 0.f;
        wf[e] = make_uint2(pack(w[0], w[1]), pack(w[2], w[3]));
    }
    const bool on_b = c0 + 4 * g < W, on_lo = c0 + 8 * t < W, on_hi = c0 + 8 * t + 4 < W;
    float4 bl = make_float4(0.f, 0.f, 0.f, 0.f), bh = bl;
    if (a.bias) {
        bl = ld4(a.bias + c0 + 8 * t, on_lo);
        bh = ld4(a.bias + c0 + 8 * t + 4, on_hi);
    }
    __syncthreads();
    for (long tile = blockIdx.x; tile < q.tiles; tile += gridDim.x) {
        const long bo = tile / q.tiles_line;
        const int i0 = (int)(tile - bo * q.tiles_line) * 16;
        const long b = bo / a.n_outer, outer = bo - b * a.n_outer;
        const float *in = a.in + b * nz * slab + outer * a.o_stride * W;
        uint32_t ba[4];  // the basis's rows of this tile
        {
            auto at = [&](int i, int k) { return i0 + i < a.n_line ? a.bas[(long)(i0 + i) * KM + k] : 0.f; };
            const int k = 4 * t;
            ba[0] = pack(at(g, k), at(g, k + 1)), ba[1] = pack(at(g + 8, k), at(g + 8, k + 1));
            ba[2] = pack(at(g, k + 2), at(g, k + 3)), ba[3] = pack(at(g + 8, k + 2), at(g + 8, k + 3));
        }
        for (int z0 = 0; z0 < nz; z0 += 32) {
            const int zn = min(32, nz - z0);
            for (int z = warp; z < zn; z += 8) {
                const float *p = a.sp + (b * nz + z0 + z) * a.sp_s + outer * a.sp_o + 4 * t * a.sp_j + c0 + 4 * g;
                float4 v[4];
#pragma unroll
                for (int j = 0; j < 4; j++) v[j] = ld4(p + j * a.sp_j, on_b);
                uint32_t bf[4][2];
                b_rows(bf, v);
                float acc[4][4] = {};
#pragma unroll
                for (int j = 0; j < 4; j++) mma(acc[j], ba, bf[j]);
                // 16-byte words of a row swapped by (depth + cell) & 1: free of
                // bank conflicts here and below
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    float4 *o = spec + (z * 16 + g + 8 * h) * 8;
                    const int f = (z + g) & 1;
                    o[(2 * t) ^ f] = acc_lo(acc, h);
                    o[(2 * t + 1) ^ f] = acc_hi(acc, h);
                }
            }
            __syncthreads();
            const int mts = zn > 16 ? 2 : 1;
#pragma unroll 1
            for (int ci = warp; ci < 16 && i0 + ci < a.n_line; ci += 8) {
                const long cell = (i0 + ci) * a.l_stride * W;
                float acc[2][4][4] = {}, dep[2][4][4] = {};
                // channel mixing: this cell's depths x channels
                const float *pc = in + (long)(z0 + g) * slab + cell + 4 * t;
#pragma unroll 2
                for (int s = 0; s < ws; s++) {
                    float4 v[4];
#pragma unroll
                    for (int r = 0; r < 4; r++)
                        v[r] = ld4(pc + 8 * r * slab + 16 * s, 16 * s + 4 * t < W && 8 * r + g < zn);
                    uint32_t bf[4][2];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const uint2 w = wf[(s * 4 + j) * 32 + lane];
                        bf[j][0] = w.x, bf[j][1] = w.y;
                    }
#pragma unroll
                    for (int m = 0; m < 2; m++) {
                        const uint32_t af[4] = {pack(v[2 * m].x, v[2 * m].y), pack(v[2 * m + 1].x, v[2 * m + 1].y),
                                                pack(v[2 * m].z, v[2 * m].w), pack(v[2 * m + 1].z, v[2 * m + 1].w)};
                        if (m < mts)
#pragma unroll
                            for (int j = 0; j < 4; j++) mma(acc[m][j], af, bf[j]);
                    }
                }
#pragma unroll
                for (int m = 0; m < 2; m++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int z = 16 * m + 8 * h + g, f = (z + ci) & 1;
                        const float4 *o = spec + (z * 16 + ci) * 8;
                        const bool on = z < zn;
                        const float4 lo = on ? o[(2 * t) ^ f] : make_float4(0, 0, 0, 0);
                        const float4 hi = on ? o[(2 * t + 1) ^ f] : make_float4(0, 0, 0, 0);
#pragma unroll
                        for (int j = 0; j < 4; j++) acc[m][j][2 * h] += comp(lo, j), acc[m][j][2 * h + 1] += comp(hi, j);
                    }
                // depth mixing: all depths of the cell
                const float *pd = in + (long)(4 * t) * slab + cell + c0 + 4 * g;
#pragma unroll 2
                for (int s = 0; s < zs; s++) {
                    float4 v[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) v[j] = ld4(pd + (16 * s + j) * slab, on_b && 16 * s + 4 * t + j < nz);
                    uint32_t bf[4][2];
                    b_rows(bf, v);
#pragma unroll
                    for (int m = 0; m < 2; m++) {
                        if (m < mts) {
                            const uint4 d4 = df[((z0 / 16 + m) * zs + s) * 32 + lane];
                            const uint32_t af[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
                            for (int j = 0; j < 4; j++) mma(dep[m][j], af, bf[j]);
                        }
                    }
                }
#pragma unroll
                for (int m = 0; m < 2; m++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int z = 16 * m + 8 * h + g;
                        if (z >= zn) continue;
                        const long o = (b * nz + z0 + z) * slab + outer * a.o_stride * W + cell + c0 + 8 * t;
                        float4 lo = acc_lo(acc[m], h), hi = acc_hi(acc[m], h);
                        const float4 dl = acc_lo(dep[m], h), dh = acc_hi(dep[m], h);
                        lo.x = lo.x + dl.x + bl.x, lo.y = lo.y + dl.y + bl.y;
                        lo.z = lo.z + dl.z + bl.z, lo.w = lo.w + dl.w + bl.w;
                        hi.x = hi.x + dh.x + bh.x, hi.y = hi.y + dh.y + bh.y;
                        hi.z = hi.z + dh.z + bh.z, hi.w = hi.w + dh.w + bh.w;
                        if (PRE) {
                            if (on_lo) *reinterpret_cast<float4 *>(a.pre + o) = lo;
                            if (on_hi) *reinterpret_cast<float4 *>(a.pre + o + 4) = hi;
                        }
                        if (ACT) {
                            lo.x = net_gelu(lo.x), lo.y = net_gelu(lo.y), lo.z = net_gelu(lo.z), lo.w = net_gelu(lo.w);
                            hi.x = net_gelu(hi.x), hi.y = net_gelu(hi.y), hi.z = net_gelu(hi.z), hi.w = net_gelu(hi.w);
                        }
                        if (on_lo) *reinterpret_cast<float4 *>(a.out + o) = lo;
                        if (on_hi) *reinterpret_cast<float4 *>(a.out + o + 4) = hi;
                    }
            }
            __syncthreads();
        }
    }
}

// -------------------------------------------------------- weight gradients
// C[m, n] += sum_r A[r, m] B[r, n] over `rows` rows of MA and NB columns, and
// colsum[n] += sum_r B[r, n]; with GELU, B is first multiplied by gelu'(pre)
// in place. One block per `chunk` rows and 32 x 32 tile of C. Of every 128
// rows, each warp loads 16 (layout `rows`) and leaves them as BF16 fragments
// in shared memory while the next ones are on their way; then it takes all
// 128 through one of the tile's eight 16 x 8 accumulators. So a block keeps
// 32 KB in flight and a sum still runs through its rows in one chain, whose
// truncations (the tensor cores' accumulators do not round) are those of one
// warp walking the same rows. The blocks' sums are added to C atomically.
constexpr int kStage = 128;

template <bool GELU>
__global__ void __launch_bounds__(256, 2) k_weight_grad(const float *__restrict__ A, int MA, float *B, int NB, long rows,
                                                        long chunk, const float *__restrict__ pre, float *C,
                                                        float *colsum) {
    __shared__ uint4 fa[2][8][2][32];
    __shared__ uint2 fb[2][8][4][32];
    __shared__ float red[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int nt = (NB + 31) / 32, m0 = (int)(blockIdx.y / nt) * 32, n0 = (int)(blockIdx.y % nt) * 32;
    const int ma = m0 + 4 * g, nb = n0 + 4 * g;
    const bool va = MA % 4 == 0, vb = NB % 4 == 0;
    const long rbeg = blockIdx.x * chunk, rend = min(rows, rbeg + chunk);
    if (tid < 32) red[tid] = 0.f;
    auto load = [&](const float *p, long r, int c, int cols, bool vec) {
        if (r >= rend) return make_float4(0.f, 0.f, 0.f, 0.f);
        p += r * cols + c;
        if (vec) return ld4(p, c < cols);
        return make_float4(c < cols ? p[0] : 0.f, c + 1 < cols ? p[1] : 0.f, c + 2 < cols ? p[2] : 0.f,
                           c + 3 < cols ? p[3] : 0.f);
    };
    float4 a[4], b[4], p[4];
    auto fetch = [&](long r) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            b[j] = load(B, r + j, nb, NB, vb);
            if (GELU) p[j] = load(pre, r + j, nb, NB, true);
            a[j] = load(A, r + j, ma, MA, va);
        }
    };
    const int mt = warp >> 2, jt = warp & 3;  // this warp's accumulator
    float acc[4] = {};
    float4 cs = make_float4(0.f, 0.f, 0.f, 0.f);
    long r = rbeg + 16 * warp + 4 * t;
    fetch(r);
    int buf = 0;
    for (long r0 = rbeg; r0 < rend; r0 += kStage, r += kStage, buf ^= 1) {
        if (GELU) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                b[j].x *= net_gelu_d(p[j].x), b[j].y *= net_gelu_d(p[j].y);
                b[j].z *= net_gelu_d(p[j].z), b[j].w *= net_gelu_d(p[j].w);
                if (r + j < rend && nb < NB) *reinterpret_cast<float4 *>(B + (r + j) * NB + nb) = b[j];
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) cs.x += b[j].x, cs.y += b[j].y, cs.z += b[j].z, cs.w += b[j].w;
        uint32_t bf[4][2];
        b_rows(bf, b);
#pragma unroll
        for (int j = 0; j < 4; j++) fb[buf][warp][j][lane] = make_uint2(bf[j][0], bf[j][1]);
        // columns 4g + 2m, 4g + 2m + 1 of A: rows g, g + 8 of tile m
#pragma unroll
        for (int m = 0; m < 2; m++)
            fa[buf][warp][m][lane] =
                make_uint4(pack(comp(a[0], 2 * m), comp(a[1], 2 * m)), pack(comp(a[0], 2 * m + 1), comp(a[1], 2 * m + 1)),
                           pack(comp(a[2], 2 * m), comp(a[3], 2 * m)), pack(comp(a[2], 2 * m + 1), comp(a[3], 2 * m + 1)));
        fetch(r + kStage);
        __syncthreads();  // two buffers: the next pass writes the other one
#pragma unroll
        for (int s = 0; s < 8; s++) {
            const uint4 a4 = fa[buf][s][mt][lane];
            const uint2 b2 = fb[buf][s][jt][lane];
            const uint32_t af[4] = {a4.x, a4.y, a4.z, a4.w}, bs[2] = {b2.x, b2.y};
            mma(acc, af, bs);
        }
    }
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const int m = m0 + 4 * g + 2 * mt + (c >> 1), n = n0 + 8 * t + 4 * (c & 1) + jt;
        if (m < MA && n < NB) atomicAdd(C + (long)m * NB + n, acc[c]);
    }
    if (m0) return;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; j++) {
        float v = comp(cs, j);
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        if (t == 0) atomicAdd(red + 4 * g + j, v);
    }
    __syncthreads();
    if (tid < 32 && n0 + tid < NB) atomicAdd(colsum + n0 + tid, red[tid]);
}

// C[z, z'] += sum over samples and the slab's columns of A[b, z] B[b, z'],
// both [batch][nz][slab]. Warps stream 32 columns of a 32 x 32 tile's rows
// (layout `cols` for both operands).
__global__ void __launch_bounds__(256, 2) k_depth_grad(const float *__restrict__ A, const float *__restrict__ B, int nz,
                                                       long slab, int batch, float *C) {
    __shared__ float red[32 * 32];
    const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int nt = (nz + 31) / 32, m0 = (int)(blockIdx.y / nt) * 32, n0 = (int)(blockIdx.y % nt) * 32;
    for (int e = tid; e < 1024; e += 256) red[e] = 0.f;
    __syncthreads();
    float acc[2][4][4] = {};
    const bool vec = slab % 4 == 0;
    auto load = [&](const float *p, long c, bool row) {
        if (vec) return ld4(p, row && c < slab);
        return make_float4(row && c < slab ? p[0] : 0.f, row && c + 1 < slab ? p[1] : 0.f,
                           row && c + 2 < slab ? p[2] : 0.f, row && c + 3 < slab ? p[3] : 0.f);
    };
    const long chunks = (slab + 31) / 32, items = chunks * batch;
    for (long it = (long)blockIdx.x * 8 + (tid >> 5); it < items; it += (long)gridDim.x * 8) {
        const long b = it / chunks, c = (it - b * chunks) * 32 + 4 * t;
        const float *pa = A + (b * nz + m0 + g) * slab + c, *pb = B + (b * nz + n0 + g) * slab + c;
        float4 x[2][4], y[2][4];
#pragma unroll
        for (int s = 0; s < 2; s++)
#pragma unroll
            for (int r = 0; r < 4; r++) {
                x[s][r] = load(pa + 8 * r * slab + 16 * s, c + 16 * s, m0 + 8 * r + g < nz);
                y[s][r] = load(pb + 8 * r * slab + 16 * s, c + 16 * s, n0 + 8 * r + g < nz);
            }
#pragma unroll
        for (int s = 0; s < 2; s++) {
            uint32_t bf[4][2];
#pragma unroll
            for (int j = 0; j < 4; j++) bf[j][0] = pack(y[s][j].x, y[s][j].y), bf[j][1] = pack(y[s][j].z, y[s][j].w);
#pragma unroll
            for (int m = 0; m < 2; m++) {
                const float4 &u = x[s][2 * m], &v = x[s][2 * m + 1];
                const uint32_t af[4] = {pack(u.x, u.y), pack(v.x, v.y), pack(u.z, u.w), pack(v.z, v.w)};
#pragma unroll
                for (int j = 0; j < 4; j++) mma(acc[m][j], af, bf[j]);
            }
        }
    }
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int c = 0; c < 4; c++)
                atomicAdd(red + (16 * m + g + 8 * (c >> 1)) * 32 + 8 * j + 2 * t + (c & 1), acc[m][j][c]);
    __syncthreads();
    for (int e = tid; e < 1024; e += 256) {
        const int m = m0 + (e >> 5), n = n0 + (e & 31);
        if (m < nz && n < nz) atomicAdd(C + (long)m * nz + n, red[e]);
    }
}

int sm_count() {
    static const int n = [] {
        int v = 0;
        EGX_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, 0));
        return v;
    }();
    return n;
}

LayerK layer_geom(const NetLayer &a) {
    LayerK q;
    q.a = a;
    q.tiles_line = (a.n_line + 15) / 16;
    q.zc = (a.nz + 31) / 32;
    q.tiles = (long)a.batch * a.n_outer * q.tiles_line;
    q.o_d = kSpecBytes;
    q.o_w = q.o_d + (uint32_t)(2 * q.zc * ((a.nz + 15) / 16)) * 512u;
    return q;
}
uint32_t layer_smem(const LayerK &q) { return q.o_w + (uint32_t)((q.a.W + 15) / 16) * 1024u; }

template <bool PRE, bool ACT>
void launch_layer(const LayerK &q, cudaStream_t s) {
    const uint32_t bytes = layer_smem(q);
    raise_smem_limit((const void *)k_layer<PRE, ACT>, bytes);
    const dim3 grid((unsigned)std::min<long>(q.tiles, (long)sm_count() * 2), (q.a.W + 31) / 32);
    k_layer<PRE, ACT><<<grid, 256, bytes, s>>>(q);
    EGX_CUDA(cudaGetLastError());
}

}  // namespace

bool net_layer_fits(int nz, int W) {
    NetLayer a{};
    a.nz = nz, a.W = W;
    return W % 4 == 0 && nz <= 1024 && layer_smem(layer_geom(a)) <= 200 * 1024;
}

void net_layer(const NetLayer &a, cudaStream_t s, long *launches) {
    const LayerK q = layer_geom(a);
    if (a.pre)
        a.act ? launch_layer<true, true>(q, s) : launch_layer<true, false>(q, s);
    else
        a.act ? launch_layer<false, true>(q, s) : launch_layer<false, false>(q, s);
    if (launches) ++*launches;
}

void net_analysis(const float *bas, int K, const float *in, long ks, long in_b, long batch, int N, float *out,
                  cudaStream_t s, long *launches) {
    const long items = batch * ((N + 31) / 32);
    const size_t bytes = (size_t)((K + 15) / 16) * 512;
    raise_smem_limit((const void *)k_analysis, bytes);
    k_analysis<<<(unsigned)std::min<long>((items + 7) / 8, (long)sm_count() * 3), 256, bytes, s>>>(bas, in, K, ks, in_b,
                                                                                                    N, items, out);
    EGX_CUDA(cudaGetLastError());
    if (launches) ++*launches;
}

void net_weight_grad(const float *A, int MA, float *B, int NB, long rows, const float *pre, float *C, float *colsum,
                     cudaStream_t s, long *launches) {
    const unsigned tiles = (unsigned)(((MA + 31) / 32) * ((NB + 31) / 32));
    // 256 chains: a block each, all of them resident at once
    const long split = std::min<long>(256, std::max<long>(1, rows / 512));
    const long chunk = ((rows + split - 1) / split + 31) / 32 * 32;
    const dim3 grid((unsigned)((rows + chunk - 1) / chunk), tiles);
    if (pre)
        k_weight_grad<true><<<grid, 256, 0, s>>>(A, MA, B, NB, rows, chunk, pre, C, colsum);
    else
        k_weight_grad<false><<<grid, 256, 0, s>>>(A, MA, B, NB, rows, chunk, nullptr, C, colsum);
    EGX_CUDA(cudaGetLastError());
    if (launches) ++*launches;
}

void net_depth_grad(const float *A, const float *B, int nz, long slab, int batch, float *C, cudaStream_t s,
                    long *launches) {
    const unsigned nt = (unsigned)((nz + 31) / 32), tiles = nt * nt;
    const long work = ((slab + 31) / 32 * batch + 7) / 8;
    const dim3 grid((unsigned)std::min<long>(work, std::max<long>(1, (long)sm_count() * 2 / tiles)), tiles);
    k_depth_grad<<<grid, 256, 0, s>>>(A, B, nz, slab, batch, C);
    EGX_CUDA(cudaGetLastError());
    if (launches) ++*launches;
}

}  // namespace egx
