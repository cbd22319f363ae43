// Instantiations of the DMMA GEMM kernel (one group of operand combinations per file, so that they
// compile in parallel).
#include "zgemm_kernel.cuh"

namespace afqmc {
namespace zg {

// A^T * B^T
int launch_tt(cudaStream_t s, int batch, const GemmParams& p, const Shape& sh) {
  return launch_tn<Op<true, false, false, true, false, false>>(s, batch, p, sh);
}

// A * conj(B)
int launch_nc(cudaStream_t s, int batch, const GemmParams& p, const Shape& sh) {
  return launch_tn<Op<false, false, false, false, true, false>>(s, batch, p, sh);
}

}  // namespace zg
}  // namespace afqmc
