// Instantiations of the DMMA GEMM kernel (one group of operand combinations per file, so that they
// compile in parallel).
#include "zgemm_kernel.cuh"

namespace afqmc {
namespace zg {

// real A * B
int launch_rn(cudaStream_t s, int batch, const GemmParams& p, const Shape& sh) {
  return launch_tn<Op<false, false, true, false, false, false>>(s, batch, p, sh);
}

}  // namespace zg
}  // namespace afqmc
