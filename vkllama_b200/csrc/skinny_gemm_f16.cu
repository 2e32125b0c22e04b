// FP16 kernels of skinny_gemm.cuh: a module of their own, loaded by the first call that needs them.
#include "skinny_gemm.cuh"

namespace vkl {

cudaError_t launch_skinny_gemm_f16(const MvParams &p, int epilogue, cudaStream_t s) { return launch_kind<false>(p, epilogue, s); }

}  // namespace vkl
