// Shapes and dispatch of the batched complex128 GEMM (zgemm.cuh; the kernel is in
// zgemm_kernel.cuh, its instantiations in zgemm_*.cu).
#include "zgemm.cuh"

namespace afqmc {
namespace zg {

using Launch = int (*)(cudaStream_t, int, const GemmParams&, const Shape&);
int launch_nn(cudaStream_t, int, const GemmParams&, const Shape&);
int launch_rn(cudaStream_t, int, const GemmParams&, const Shape&);
int launch_nr(cudaStream_t, int, const GemmParams&, const Shape&);
int launch_nt(cudaStream_t, int, const GemmParams&, const Shape&);
int launch_nrt(cudaStream_t, int, const GemmParams&, const Shape&);
int launch_tt(cudaStream_t, int, const GemmParams&, const Shape&);
int launch_tn(cudaStream_t, int, const GemmParams&, const Shape&);
int launch_hn(cudaStream_t, int, const GemmParams&, const Shape&);
int launch_rrt(cudaStream_t, int, const GemmParams&, const Shape&);
int launch_nc(cudaStream_t, int, const GemmParams&, const Shape&);
int launch_nh(cudaStream_t, int, const GemmParams&, const Shape&);
int launch_rtn(cudaStream_t, int, const GemmParams&, const Shape&);
int launch_nrt_sym(cudaStream_t, const GemmParams&, const Shape&);

namespace {

constexpr int SMS = 148;

// Columns of a tile in units of 8, at most 8 of them: the number that pads n least, where a
// narrower tile has to save 1/32 of the work per unit given up (it reads A that much more often).
int fit_cols(int n) {
  const int need = ceil_div(n, 8);
  if (need <= 8) return need;
  int best = 8;
  long cost = long(ceil_div(need, 8)) * 8 * 32;
  for (int c = 7; c >= 4; --c) {
    const long q = long(ceil_div(need, c)) * c * (32 + 8 - c);
    if (q < cost) {
      cost = q;
      best = c;
    }
  }
  return best;
}

// Warps (8-row strips) of a tile.  The FP64 tensor path belongs to the SM's four schedulers, and a
// CTA's warp i runs on scheduler i mod 4 whatever else is resident: 5 strips take the time of 8
// (m=200, n=50, k=200, 1024 problems: 813 us with 5 warps, which divide 200, 678 us with 4,
// 749 us with 8).  So strips count in groups of four; four warps read B twice as often as eight,
// which costs them about 1/16.
int fit_rows(int m) {
  const int need = ceil_div(m, 8);
  if (need <= 8) return need;
  const long four = long(ceil_div(need, 4)) * 4 * 17, eight = long(ceil_div(need, 8)) * 8 * 16;
  if (four < eight) return 4;
  for (int w = 5; w < 8; ++w)  // the same number of tiles with less padding to load
    if (ceil_div(need, w) == ceil_div(need, 8)) return w;
  return 8;
}

}  // namespace

// The CTA shape: tiles fitted to m and n; then, where those are too few to give every SM one, the
// K range of a single problem split over a cluster of up to 8 CTAs (each keeping at least 8 K
// tiles, so that the reduction stays small against the product), and the tiles halved down to 8
// strips in all (below that the operand loads bound a tile).
Shape shape(int batch, int m, int n, int k) {
  Shape sh{fit_rows(m), fit_cols(n), 1};
  auto ctas = [&] { return long(ceil_div(m, 8 * sh.warps)) * ceil_div(n, 8 * sh.tn) * batch; };
  if (batch == 1 && ctas() < SMS) {
    const long s = SMS / ctas(), ks = ceil_div(k, 16) / 8;
    const long c = s < ks ? s : ks;
    sh.split = int(c < 1 ? 1 : (c > 8 ? 8 : c));
  }
  while (ctas() * sh.split < SMS && sh.warps * sh.tn > 8) {
    if (sh.tn >= sh.warps)
      sh.tn = (sh.tn + 1) / 2;
    else
      sh.warps = (sh.warps + 1) / 2;
  }
  if (m > 65535l * 8 * sh.warps) sh.warps = 8;  // grid.y limit
  return sh;
}

}  // namespace zg

int zgemm(cudaStream_t s, int batch, GemmTrans ta, bool a_real, GemmTrans tb, bool b_real,
          const GemmParams& p) {
  if (p.m <= 0 || p.n <= 0 || batch <= 0) return AFQMC_OK;
  if (p.k <= 0) {
    set_error_detail("zgemm: k = 0 is not supported by the kernel launcher");
    return AFQMC_ERR_SHAPE;
  }
  if (batch > 65535) {
    set_error_detail("zgemm: batch %d exceeds the grid limit", batch);
    return AFQMC_ERR_SHAPE;
  }
  const bool AT = (ta == GT || ta == GH), AC = (ta == GC || ta == GH);
  const bool BT = (tb == GT || tb == GH), BC = (tb == GC || tb == GH);
  if ((a_real && AC) || (b_real && BC)) {
    // conjugating a real operand is the identity
    return zgemm(s, batch, AT ? GT : GN, a_real, BT ? GT : GN, b_real, p);
  }
  // Instantiated combinations (the products the walker step and its setup use).
  zg::Launch fn = nullptr;
#define AFQMC_GEMM_CASE(at, ac, ar, bt, bc, br, name) \
  if (AT == at && AC == ac && a_real == ar && BT == bt && BC == bc && b_real == br) fn = zg::name;
  AFQMC_GEMM_CASE(false, false, false, false, false, false, launch_nn)  // A*B
  AFQMC_GEMM_CASE(false, false, true, false, false, false, launch_rn)   // real A * B
  AFQMC_GEMM_CASE(false, false, false, false, false, true, launch_nr)   // A * real B
  AFQMC_GEMM_CASE(false, false, false, true, false, false, launch_nt)   // A * B^T
  AFQMC_GEMM_CASE(false, false, false, true, false, true, launch_nrt)   // A * real B^T
  AFQMC_GEMM_CASE(true, false, false, true, false, false, launch_tt)    // A^T * B^T
  AFQMC_GEMM_CASE(true, false, false, false, false, false, launch_tn)   // A^T * B
  AFQMC_GEMM_CASE(true, false, true, false, false, false, launch_rtn)   // real A^T * B
  AFQMC_GEMM_CASE(true, true, false, false, false, false, launch_hn)    // A^H * B
  AFQMC_GEMM_CASE(false, false, true, true, false, true, launch_rrt)    // real A * real B^T
  AFQMC_GEMM_CASE(false, false, false, false, true, false, launch_nc)   // A * conj(B)
  AFQMC_GEMM_CASE(false, false, false, true, true, false, launch_nh)    // A * B^H
#undef AFQMC_GEMM_CASE
  if (!fn) {
    set_error_detail(
        "zgemm: operand combination (ta=%d a_real=%d tb=%d b_real=%d) not instantiated", int(ta),
        int(a_real), int(tb), int(b_real));
    return AFQMC_ERR_UNSUPPORTED;
  }
  return fn(s, batch, p, zg::shape(batch, p.m, p.n, p.k));
}

int zgemm_sym_pairs(cudaStream_t s, int M, const GemmParams& p) {
  if (p.m <= 0 || M <= 0) return AFQMC_OK;
  GemmParams q = p;
  q.sym_m = M;
  q.n = M * M;
  // Worth it once the blocks fill the SMs twice over: below that the time is one tile's, and the
  // general form's tiles can be narrower than the 64 pairs of a block.  (1024 walkers, M = 200,
  // 1600 vectors: 4.73 ms, against 8.6 ms for all pairs.)
  const long nb = ceil_div(M, 8), blocks = nb * (nb + 1) / 2;
  if (ceil_div(p.m, 64) * blocks < 2 * zg::SMS) return zgemm(s, 1, GN, false, GT, true, q);
  zg::Shape sh{zg::fit_rows(p.m), 8, 1};
  if (p.m > 65535l * 8 * sh.warps) sh.warps = 8;
  return zg::launch_nrt_sym(s, q, sh);
}

}  // namespace afqmc
