// Instantiations of the DMMA GEMM kernel (one group of operand combinations per file, so that they
// compile in parallel).
#include "zgemm_kernel.cuh"

namespace afqmc {
namespace zg {

// A * real B
int launch_nr(cudaStream_t s, int batch, const GemmParams& p, const Shape& sh) {
  return launch_tn<Op<false, false, false, false, false, true>>(s, batch, p, sh);
}

// real A * real B^T
int launch_rrt(cudaStream_t s, int batch, const GemmParams& p, const Shape& sh) {
  return launch_tn<Op<false, false, true, true, false, true>>(s, batch, p, sh);
}

}  // namespace zg
}  // namespace afqmc
