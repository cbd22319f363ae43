// Batched re-orthonormalisation of the walkers' Slater matrices.
//
// Reference: det_ops::orthogonalize (src/AFQMC/SlaterDeterminantOperations/orthogonalize.hpp:
// 131-169) calls LAPACK geqrf + ungqr on each S_w (M x N) and multiplies column i of Q by
// scl_i = sign(Re R_ii) (log_determinant_from_geqrf, numerics/operations/determinants_impl.hpp:
// 77-108).  The result is the unique Q whose R has a real positive diagonal, so any stable QR gives
// the same walker.  Here: CholeskyQR2 — the Gram matrices S^H S and the products S R^{-1} run as
// batched DMMA GEMMs, the N x N Cholesky factorisations and triangular inverses in one CTA per
// walker; two passes make Q orthonormal to rounding for the well-conditioned matrices that periodic
// re-orthogonalisation keeps.
#include "detops.cuh"
#include "dmma.cuh"
#include "zgemm.cuh"

namespace afqmc {
namespace {

// ---------------------------------------------------------------------------------------------
// CholeskyQR: G = S^H S = R^H R (R upper, real positive diagonal), Rinv = R^{-1}; one CTA of four
// warps per walker, eight rows at a time.  logdetR[w] += sum_i log R_ii.
//
// Right-looking elimination of [G | I]: with R11^H R11 the panel's 8 x 8 diagonal block,
//   rows K     <- R11^{-H} rows K
//   rows below -= R[K, i]^H rows K
// turns G into R and the identity into R^{-H}, whose conjugate transpose is the result.  One array
// holds both: R only feeds the trailing update of its own panel, so R^{-H} (lower triangular)
// takes the diagonal blocks as they finish and the blocks below them.  The 8 x 8 block is one
// warp's work (a column per lane, rows by shuffle); the rest are rank-8 updates on the FP64 tensor
// path.  The array is padded to a multiple of 8 with an identity block.
// Bound by the chain of 8 x 8 factorisations and the barriers between; four CTAs fit an SM at
// N = 50.  1024 walkers, N = 50: the form with a barrier per row and a serial back substitution
// per column took 396 us, this one 81.
// ---------------------------------------------------------------------------------------------
constexpr int CH_THREADS = 128;

constexpr int CH_MAX_N = 85;  // the largest N that orthogonalize takes (shared memory holds 112)

__host__ __device__ inline int ch_pad(int N) { return (N + 7) / 8 * 8; }
inline size_t ch_smem(int N) { return size_t(ch_pad(N)) * (ch_pad(N) + 1) * sizeof(c128); }

__global__ void __launch_bounds__(CH_THREADS, 4)
    chol_inv_kernel(const c128* __restrict__ Gram, c128* __restrict__ Rinv, c128* __restrict__ logdetR,
                    int N) {
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double dg[128];  // R_ii
  c128* a = reinterpret_cast<c128*>(smem_raw);  // [N8][P]
  const int N8 = ch_pad(N), P = N8 + 1, NT = N8 / 8;
  const long w = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const c128* Gw = Gram + w * long(N) * N;
  for (int e = tid; e < N8 * N8; e += CH_THREADS) {
    const int i = e / N8, j = e - i * N8;
    c128 v = cmk(i == j ? 1.0 : 0.0, 0.0);
    if (i < N && j < N) v = (i / 8 <= j / 8) ? Gw[long(i) * N + j] : cmk(0.0, 0.0);
    a[i * P + j] = v;
  }
  __syncthreads();

  for (int kt = 0; kt < NT; ++kt) {
    const int k0 = 8 * kt;
    if (warp == 0) {
      // lanes 0..7: column `lane` of the diagonal block; lanes 8..15: column lane - 8 of the
      // identity, which becomes R11^{-H}; the other lanes follow lanes 0..15
      const int c = lane & 7;
      const bool inv = (lane & 8) != 0;
      c128 v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        v[i] = inv ? cmk(i == c ? 1.0 : 0.0, 0.0) : a[(k0 + i) * P + k0 + c];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        double d = __shfl_sync(FULL, v[j].x, j);
        d = d > 1e-300 ? sqrt(d) : 1e-150;
        const double dinv = 1.0 / d;
        if (lane == 0) dg[k0 + j] = d;
        v[j] = cscale(v[j], dinv);
#pragma unroll
        for (int i = j + 1; i < 8; ++i) {
          // R[j][i], lane i's element j
          const c128 rji = cmk(__shfl_sync(FULL, v[j].x, i), -__shfl_sync(FULL, v[j].y, i));
          v[i] = csub(v[i], cmul(rji, v[j]));
        }
      }
      if (lane >= 8 && lane < 16)
#pragma unroll
        for (int i = 0; i < 8; ++i) a[(k0 + i) * P + k0 + c] = v[i];
    }
    __syncthreads();
    // rows K of every other column block: R11^{-H} times them (a warp owns a block)
    for (int tj = warp; tj < NT; tj += CH_THREADS / 32) {
      if (tj == kt) continue;
      double cr[2] = {0.0, 0.0}, ci[2] = {0.0, 0.0};
#pragma unroll
      for (int kk = 0; kk < 8; kk += 4)
        zmma(cr, ci, a[(k0 + g) * P + k0 + kk + t], a[(k0 + kk + t) * P + tj * 8 + g]);
      __syncwarp();
#pragma unroll
      for (int h = 0; h < 2; ++h) a[(k0 + g) * P + tj * 8 + 2 * t + h] = cmk(cr[h], ci[h]);
    }
    __syncthreads();
    // rows below: the upper blocks of what is left of G, and R^{-H}'s blocks up to the panel
    const int below = NT - 1 - kt;
    for (int e = warp; e < below * NT; e += CH_THREADS / 32) {
      const int tj = e / below, ti = kt + 1 + (e - tj * below);
      if (tj > kt && tj < ti) continue;
      double cr[2], ci[2];
      c128* dst = a + (ti * 8 + g) * P + tj * 8 + 2 * t;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const c128 v = dst[h];
        cr[h] = v.x;
        ci[h] = v.y;
      }
#pragma unroll
      for (int kk = 0; kk < 8; kk += 4) {
        const c128 r = a[(k0 + kk + t) * P + ti * 8 + g];  // - conj(R[K][i])
        zmma(cr, ci, cmk(-r.x, r.y), a[(k0 + kk + t) * P + tj * 8 + g]);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) dst[h] = cmk(cr[h], ci[h]);
    }
    __syncthreads();
  }
  c128* Rw = Rinv + w * long(N) * N;
  for (int e = tid; e < N * N; e += CH_THREADS) {
    const int i = e / N, j = e - i * N;
    Rw[e] = i <= j ? cconj(a[j * P + i]) : cmk(0.0, 0.0);
  }
  if (warp == 0) {
    double sr = 0.0;
    for (int i = lane; i < N; i += 32) sr += log(dg[i]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sr += __shfl_xor_sync(FULL, sr, off);
    if (lane == 0) logdetR[w] = cadd(logdetR[w], cmk(sr, 0.0));
  }
}

}  // namespace

// One CholeskyQR pass: Q = S R^{-1} written to Q (ldQ), R from the Gram matrix of S.
static int cholqr_pass(cudaStream_t s, const c128* S, long ldS, c128* Q, long ldQ, c128* logdetR,
                       int W, int M, int N, c128* gram, c128* rinv) {
  GemmParams g{};
  g.m = N; g.n = N; g.k = M;
  g.A = S; g.lda = N; g.strideA = ldS;  // A^H with A stored [M][N]
  g.B = S; g.ldb = N; g.strideB = ldS;
  g.C = gram; g.ldc = N; g.strideC = long(N) * N;
  g.alpha = cmk(1, 0); g.beta = cmk(0, 0);
  AFQMC_TRY(zgemm(s, W, GH, false, GN, false, g));
  const size_t smem = ch_smem(N);
  AFQMC_TRY(allow_smem(chol_inv_kernel, smem, ch_smem(CH_MAX_N)));
  chol_inv_kernel<<<W, CH_THREADS, smem, s>>>(gram, rinv, logdetR, N);
  AFQMC_TRY(launch_status("chol_inv_kernel"));
  GemmParams q{};
  q.m = M; q.n = N; q.k = N;
  q.A = S; q.lda = N; q.strideA = ldS;
  q.B = rinv; q.ldb = N; q.strideB = long(N) * N;
  q.C = Q; q.ldc = N; q.strideC = ldQ;
  q.alpha = cmk(1, 0); q.beta = cmk(0, 0);
  return zgemm(s, W, GN, false, GN, false, q);
}

// det_ops::orthogonalize by CholeskyQR2: two passes give Q orthonormal to rounding for the
// well-conditioned walkers that the periodic re-orthogonalisation keeps; R = R2 R1 has a real
// positive diagonal, so Q is the same unique factor as geqrf + ungqr + sign fix.
int orthogonalize(cudaStream_t s, c128* S, long ldS, c128* logdetR, int W, int M, int N,
                  c128* work) {
  if (W <= 0 || N <= 0 || M <= 0) return AFQMC_OK;
  if (N > M) {
    set_error_detail("orthogonalize: N = %d > M = %d", N, M);
    return AFQMC_ERR_SHAPE;
  }
  if (N > CH_MAX_N) {
    set_error_detail("orthogonalize: N = %d > %d", N, CH_MAX_N);
    return AFQMC_ERR_UNSUPPORTED;
  }
  const size_t nQ = size_t(W) * M * N, nG = size_t(W) * N * N;
  void* buf = work;
  if (!buf) AFQMC_CUDA_TRY(cudaMallocAsync(&buf, sizeof(c128) * (nQ + 2 * nG), s));
  c128* Q = static_cast<c128*>(buf);
  c128* gram = Q + nQ;
  c128* rinv = gram + nG;
  int st = cholqr_pass(s, S, ldS, Q, long(M) * N, logdetR, W, M, N, gram, rinv);
  if (!st) st = cholqr_pass(s, Q, long(M) * N, S, ldS, logdetR, W, M, N, gram, rinv);
  if (!work) cudaFreeAsync(buf, s);
  return st;
}

}  // namespace afqmc
