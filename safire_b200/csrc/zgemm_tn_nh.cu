// Instantiations of the DMMA GEMM kernel (one group of operand combinations per file, so that they
// compile in parallel).
#include "zgemm_kernel.cuh"

namespace afqmc {
namespace zg {

// A^T * B
int launch_tn(cudaStream_t s, int batch, const GemmParams& p, const Shape& sh) {
  return launch_tn<Op<true, false, false, false, false, false>>(s, batch, p, sh);
}

// real A^T * B
int launch_rtn(cudaStream_t s, int batch, const GemmParams& p, const Shape& sh) {
  return launch_tn<Op<true, false, true, false, false, false>>(s, batch, p, sh);
}

// A * B^H
int launch_nh(cudaStream_t s, int batch, const GemmParams& p, const Shape& sh) {
  return launch_tn<Op<false, false, false, true, true, false>>(s, batch, p, sh);
}

}  // namespace zg
}  // namespace afqmc
