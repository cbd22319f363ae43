// Shapes and dispatch of the batched complex128 GEMM (zgemm.cuh; the kernel is in
// zgemm_kernel.cuh, its instantiations in zgemm_*.cu).
#include "zgemm.cuh"

#include <algorithm>

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

// Time (cycles) of a single problem in a shape, up to what all shapes share.  A K tile of a CTA costs its
// SM the DMMAs of the busiest scheduler and the fragment loads of all its warps (x), and takes no less
// than the latency of a stage, which grows with the copies a thread issues for it; resident CTAs
// overlap that latency, and what does not fit a wave adds another; a wave fills its ring first.  Clusters
// of four and eight leave about a twelfth of the SMs unused.  The constants are fitted to timings of 114
// problems in all shapes (1..2400 rows, 26..40000 columns, K = 35..4290; 61 of them from the steps and
// energies of molecules and model systems).
double model_time(const Shape& sh, int m, int n, int k, bool a_real, bool b_real) {
  const int w = sh.warps, tn = sh.tn, c = sh.split;
  const int frag_a = a_real ? 2 : 4, frag_b = b_real ? 2 : 4;  // wavefronts of a fragment load
  const int mma = a_real && b_real ? 1 : (a_real || b_real ? 2 : 4);
  const double x = 0.6 * ((w + 3) / 4 * tn * 4 * mma * 16) + 1.6 * (w * 4 * (frag_a + tn * frag_b));
  const double latency = 90.0 * (4 + (4 * tn + w - 1) / w) + 0.9 * x;
  const int ring = STAGES * 8 * (BK + 4) * (w * (a_real ? 8 : 16) + tn * (b_real ? 8 : 16));
  const int smem = (c > 1 ? std::max(ring, 64 * w * tn * 16) : ring) + 1024;
  const int resident = std::max(1, std::min(227 * 1024 / smem, 16 / w));
  const int tiles = (m + 8 * w - 1) / (8 * w) * ((n + 8 * tn - 1) / (8 * tn));
  const int sms = c > 2 ? NUM_SMS * 11 / 12 : NUM_SMS, per_sm = (tiles * c + sms - 1) / sms;
  const int waves = per_sm / resident, rest = per_sm - waves * resident;
  const double cycles = waves * std::max(resident * x, latency) +
                        (rest ? std::max(rest * x, latency) : 0.0);
  const int ktiles = ((k + BK - 1) / BK + c - 1) / c;
  return cycles * (ktiles + STAGES - 1) + (c > 1 ? 3000.0 : 0.0);
}

// 64 x 64 tiles fill the SMs twice over
bool many_tiles(int m, long n) { return ceil_div(m, 64) * long(ceil_div(n, 64)) >= 2 * NUM_SMS; }

// The shape for a single problem of few tiles: the fitted one, or that of least time by the model if its
// time is below `worth` of the fitted shape's.  K is split in two K tiles or more each, and not where
// there are many tiles.  On the problems above the choice is within 7.5% of the fastest of all shapes in
// the mean, and never more than 1.5% slower than the fitted shape, which alone takes 1.35 times the
// fastest in the mean: 1024 x 400 x 4160 (real B) in tiles of 64 x 40 is 160 CTAs, two on 12 of the SMs
// and one on the others (462 us; in 32 x 32 333), and 1 x 4096 x 200 one warp an SM (27.5 us; in 16 x 8
// 11).  More widths than these four cost the host time (0.6 us for four) and gain 1%.
Shape least_time(Shape fit, double worth, int m, int n, int k, bool a_real, bool b_real) {
  const int ktiles = ceil_div(k, BK);
  const bool may_split = !many_tiles(m, n);
  double least = worth * model_time(fit, m, n, k, a_real, b_real);
  for (int w = m >= 64 ? 4 : 1; w <= 8 && (w <= 2 || m > 4 * w); w *= 2)
    for (const int tn : {1, 2, 4, 7}) {
      if (n <= 8 * (tn - 1)) break;
      for (int c = 1; c <= 8 && (c == 1 || (may_split && ktiles >= 2 * c)); c *= 2) {
        const double t = model_time({w, tn, c}, m, n, k, a_real, b_real);
        if (t < least) {
          least = t;
          fit = {w, tn, c};
        }
      }
    }
  return fit;
}

}  // namespace

// The CTA shape: tiles fitted to m and n; then, where those are too few to give every SM one, the K
// range of a single problem split over a cluster of up to 8 CTAs (each keeping at least 8 K tiles),
// and the tiles halved down to 8 strips in all (below that the operand loads bound a tile).  For a
// single problem of few tiles the model looks for a faster one, by a twentieth; where the fitted tiles
// give every SM two the waves cost less, and the gain has to stand out of the model's error (1024 x
// 1600 x 10000, a force bias of the M = 200 system, was 2% slower in the tiles that it put at 0.93).
Shape shape(int batch, int m, int n, int k, bool a_real, bool b_real) {
  Shape sh{fit_rows(m), fit_cols(n), 1};
  auto ctas = [&] { return long(ceil_div(m, 8 * sh.warps)) * ceil_div(n, 8 * sh.tn) * batch; };
  const bool few = batch == 1 && ctas() < 5 * NUM_SMS;
  const double worth = ctas() < 2 * NUM_SMS ? 0.95 : 0.85;
  if (batch == 1 && ctas() < NUM_SMS)
    sh.split = std::max(1, std::min({8, int(NUM_SMS / ctas()), ceil_div(k, BK) / 8}));
  while (ctas() * sh.split < NUM_SMS && sh.warps * sh.tn > 8) {
    if (sh.tn >= sh.warps)
      sh.tn = (sh.tn + 1) / 2;
    else
      sh.warps = (sh.warps + 1) / 2;
  }
  if (few) return least_time(sh, worth, m, n, k, a_real, b_real);
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
  return fn(s, batch, p, zg::shape(batch, p.m, p.n, p.k, a_real, b_real));
}

int zgemm_sym_pairs(cudaStream_t s, int M, const GemmParams& p) {
  if (p.m <= 0 || M <= 0) return AFQMC_OK;
  GemmParams q = p;
  q.sym_m = M;
  q.n = M * M;
  // Worth it where the general form has many tiles (and does not split its sums): with fewer the time
  // is one tile's, and the general form's can be narrower than the 64 pairs of a block.  Rows for
  // fewer than four warps leave a block to the latency of its loads, so two blocks an SM then.
  // (1024 walkers, M = 200, 1600 vectors: 4.73 ms, against 8.6 ms for all pairs.)
  const long nb = ceil_div(M, 8), blocks = nb * (nb + 1) / 2;
  if (!zg::many_tiles(p.m, long(M) * M) || (p.m <= 24 && blocks < 2 * NUM_SMS))
    return zgemm(s, 1, GN, false, GT, true, q);
  zg::Shape sh{zg::fit_rows(p.m), 8, 1};
  if (p.m > 65535l * 8 * sh.warps) sh.warps = 8;
  return zg::launch_nrt_sym(s, q, sh);
}

}  // namespace afqmc
