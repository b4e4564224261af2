// Learned flexible preconditioner: a spectral network on the anomaly mesh
// (declarations shared by egx_learn.cu and the solver in egx_api.cu).
#pragma once

#include "egx_common.cuh"

struct egx_net;

namespace egx {

// z = v + rms(v) N(v / rms(v)) for `batch` complex64 vectors [batch][N] on
// the device (N = nx ny 3 nz in the anomaly layout), on stream s. Uses the
// log-conductivity set by egx_net_set_model.
void net_apply(egx_net *net, const float2 *v, float2 *z, int batch, cudaStream_t s, long *launches);

// nx ny 3 nz: the vector length the network was built for
long net_length(const egx_net *net);

// Pointwise GEMM on the tcgen05 tensor cores (egx_learn_tc.cu): C[m, n] =
// sum_k A[m, k] B[k b_k + n b_n] (+ C[m, n] with accumulate) (+ bias[n] if not
// null), A row-major [M x K], C row-major [M x N], K and N in 1..32, BF16 operands, FP32
// accumulation; err receives EGX_ERR_TIMEOUT if a bounded wait expires.
bool pw_gemm_tc_fits(int K, int N);
void pw_gemm_tc(const float *A, int M, int K, const float *B, long b_k, long b_n, int N, float *C, bool accumulate,
                const float *bias, int *err, cudaStream_t s);

constexpr int kNetModes = 16;  // retained modes per lateral direction

__device__ __forceinline__ float net_gelu(float x) {
    const float c = 0.7978845608028654f;  // sqrt(2/pi)
    return 0.5f * x * (1.f + tanhf(c * (x + 0.044715f * x * x * x)));
}
__device__ __forceinline__ float net_gelu_d(float x) {
    const float c = 0.7978845608028654f;
    const float u = c * (x + 0.044715f * x * x * x), th = tanhf(u);
    return 0.5f * (1.f + th) + 0.5f * x * (1.f - th * th) * c * (1.f + 3.f * 0.044715f * x * x);
}

// A layer's three branches in one pass (egx_learn_layer.cu), for activations
// [batch][nz][ncell][W], cell = outer o_stride + i l_stride, i < n_line along
// the basis bas [n_line][modes]; D(z, z') = D[z d_o + z' d_i], Wt(k, c) =
// Wt[k w_k + c w_n], sp at (sample nz + z) sp_s + outer sp_o + mode sp_j + c.
// Writes pre = sums + bias (null: not kept) and out = act ? gelu(pre) : pre.
struct NetLayer {
    const float *in, *sp, *bas, *D, *Wt, *bias;
    float *pre, *out;
    long d_o, d_i, w_k, w_n, sp_s, sp_o, sp_j, ncell, o_stride, l_stride;
    int batch, nz, W, n_outer, n_line;
    bool act;
};
// W a multiple of 4 (16-byte loads) and the mixing weights in shared memory;
// the kernels below take W under the same rule
bool net_layer_fits(int nz, int W);
void net_layer(const NetLayer &a, cudaStream_t s, long *launches);
// out[b][i][n] = sum_k bas[k][i] in[b in_b + k ks + n], i < modes, n < N
void net_analysis(const float *bas, int K, const float *in, long ks, long in_b, long batch, int N, float *out,
                  cudaStream_t s, long *launches);
// C[m][n] += sum_r A[r][m] B[r][n], colsum[n] += sum_r B[r][n]; with pre (MA
// <= 32, NB a multiple of 4) B is first multiplied by gelu'(pre) in place
void net_weight_grad(const float *A, int MA, float *B, int NB, long rows, const float *pre, float *C, float *colsum,
                     cudaStream_t s, long *launches);
// C[z][z'] += sum over samples and columns of A[b][z] B[b][z']
void net_depth_grad(const float *A, const float *B, int nz, long slab, int batch, float *C, cudaStream_t s,
                    long *launches);

}  // namespace egx
