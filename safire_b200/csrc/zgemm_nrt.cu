// Instantiations of the DMMA GEMM kernel (one group of operand combinations per file, so that they
// compile in parallel).
#include "zgemm_kernel.cuh"

namespace afqmc {
namespace zg {

// A * real B^T
int launch_nrt(cudaStream_t s, int batch, const GemmParams& p, const Shape& sh) {
  return launch_tn<Op<false, false, false, true, false, true>>(s, batch, p, sh);
}

// A * real B^T over the pairs of a symmetric tensor
int launch_nrt_sym(cudaStream_t s, const GemmParams& p, const Shape& sh) {
  return launch<8, Op<false, false, false, true, false, true>, true>(s, 1, p, sh);
}

}  // namespace zg
}  // namespace afqmc
