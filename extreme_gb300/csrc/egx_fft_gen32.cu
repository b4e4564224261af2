// The generic transform's complex64 kernels.
#include "egx_fft_gen_kernels.cuh"

namespace egx {

EGX_GEN_INST(float)

}  // namespace egx
