// S_w <- P1 sum_{n <= order} (i V_w)^n / n! P1 S_w in complex128, one launch for all order + 2
// products of every walker (propagate.hpp:41-70, 238-298), for the sizes whose walker fits an SM.
//
// One CTA per walker.  The current term T lives in shared memory as the B operand, the running
// sum R beside it (or in registers); a warp owns SPW 8-row strips of all columns, so a strip of
// V is read by one warp only and comes straight from global memory as DMMA fragments, no staging
// and no barrier inside a product: two barriers per term.  M <= 32 keeps V's fragments in
// registers for all terms.  The sums run in the order of zgemm's, bit for bit.
//
// Against the order + 2 GEMM launches this replaces it saves the launches and their tails and the
// passes of T and R through global memory; what bounds it is the FP64 tensor path, and with few
// walkers an SM the latency of one walker's chain.  Whole steps with the launches and with this:
// M = 32, N = 8, 64 walkers 102 -> 77 us; M = 19, N = 3, 1536 walkers, two spins 619 -> 511 us;
// M = 100, N = 25, 256 walkers 708 -> 640 us.  Past N = 32 or M = 128 the accumulators and T, R
// no longer fit beside enough warps, and the products are large enough for GEMM launches; where these
// are faster below that, taylor_c128_fits tells.
#include <type_traits>

#include "detops.cuh"
#include "dmma.cuh"

namespace afqmc {
namespace {

// row pitch of T: 2 past a multiple of 8, conflict-free fragment loads
__host__ __device__ inline int t_pitch(int TN) { return 8 * TN + 2; }

// products of one warp's strips: acc[s][j] = A[strip s] (op) T.  A: M x M row-major (real or
// complex), rows and columns past M read as zero.
template <int SPW, int TN, typename TA>
struct Strips {
  double cr[SPW][TN][2], ci[SPW][TN][2];

  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int s = 0; s < SPW; ++s)
#pragma unroll
      for (int j = 0; j < TN; ++j)
        cr[s][j][0] = cr[s][j][1] = ci[s][j][0] = ci[s][j][1] = 0.0;
  }
  __device__ __forceinline__ void step(const TA (&fa)[SPW], const c128* T, int k, int g) {
    constexpr int PT = 8 * TN + 2;
    c128 fb[TN];
#pragma unroll
    for (int j = 0; j < TN; ++j) fb[j] = T[k * PT + j * 8 + g];
#pragma unroll
    for (int s = 0; s < SPW; ++s) {
      if constexpr (sizeof(TA) == 8) {
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          dmma(cr[s][j][0], cr[s][j][1], fa[s], fb[j].x);
          dmma(ci[s][j][0], ci[s][j][1], fa[s], fb[j].y);
        }
      } else {
        const double nai = -fa[s].y;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          dmma(cr[s][j][0], cr[s][j][1], fa[s].x, fb[j].x);
          dmma(ci[s][j][0], ci[s][j][1], fa[s].x, fb[j].y);
        }
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          dmma(cr[s][j][0], cr[s][j][1], nai, fb[j].y);
          dmma(ci[s][j][0], ci[s][j][1], fa[s].y, fb[j].x);
        }
      }
    }
  }
};

template <typename TA>
__device__ __forceinline__ TA zero_of();
template <>
__device__ __forceinline__ double zero_of<double>() { return 0.0; }
template <>
__device__ __forceinline__ c128 zero_of<c128>() { return cmk(0.0, 0.0); }

// the whole product, A streamed from global memory four fragments ahead
template <int SPW, int TN, typename TA>
__device__ __forceinline__ void product(Strips<SPW, TN, TA>& st, const TA* __restrict__ A,
                                        const c128* T, int M, int row0, int g, int t) {
  constexpr int PF = 4;
  st.clear();
  TA fa[2][PF][SPW];
  const TA* rows[SPW];
  bool ok[SPW];
#pragma unroll
  for (int s = 0; s < SPW; ++s) {
    const int r = row0 + 8 * s + g;
    ok[s] = r < M;
    rows[s] = A + long(ok[s] ? r : 0) * M;
  }
  auto load = [&](TA (&f)[PF][SPW], int k0) {
#pragma unroll
    for (int q = 0; q < PF; ++q)
#pragma unroll
      for (int s = 0; s < SPW; ++s) {
        const int k = k0 + 4 * q + t;
        f[q][s] = (ok[s] && k < M) ? __ldg(rows[s] + k) : zero_of<TA>();
      }
  };
  load(fa[0], 0);
  for (int k0 = 0; k0 < M; k0 += 8 * PF) {
    load(fa[1], k0 + 4 * PF);
#pragma unroll
    for (int q = 0; q < PF; ++q)
      if (k0 + 4 * q < M) st.step(fa[0][q], T, k0 + 4 * q + t, g);
    load(fa[0], k0 + 8 * PF);
#pragma unroll
    for (int q = 0; q < PF; ++q)
      if (k0 + 4 * PF + 4 * q < M) st.step(fa[1][q], T, k0 + 4 * PF + 4 * q + t, g);
  }
}

// KV > 0: V's fragments (KV of them, K = 4 KV >= M) stay in registers
template <int SPW, int TN, int KV, bool P1_REAL>
__global__ void __launch_bounds__(256, (SPW * TN <= 4 && KV == 0) ? 2 : 1)
    taylor_c128_kernel(const void* __restrict__ P1v, const c128* __restrict__ V, long strideV,
                       c128* S, long ldS, int M, int N, int order) {
  using T1 = typename std::conditional<P1_REAL, double, c128>::type;
  constexpr int PT = 8 * TN + 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int K4 = (M + 3) / 4 * 4;
  c128* T = reinterpret_cast<c128*>(smem_raw);  // [K4][PT]
  c128* R = T + size_t(K4) * PT;                // [M][8 TN]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3, row0 = warp * 8 * SPW;
  const long w = blockIdx.x;
  const T1* P1 = static_cast<const T1*>(P1v);
  const c128* Vw = V + w * strideV;
  c128* Sw = S + w * ldS;

  c128 fv[KV > 0 ? KV : 1][SPW];
  if constexpr (KV > 0) {
#pragma unroll
    for (int q = 0; q < KV; ++q)
#pragma unroll
      for (int s = 0; s < SPW; ++s) {
        const int r = row0 + 8 * s + g, k = 4 * q + t;
        fv[q][s] = (r < M && k < M) ? __ldg(Vw + long(r) * M + k) : cmk(0.0, 0.0);
      }
  }
  for (int e = tid; e < K4 * PT; e += blockDim.x) {
    const int i = e / PT, j = e - i * PT;
    T[e] = (i < M && j < N) ? Sw[long(i) * N + j] : cmk(0.0, 0.0);
  }
  __syncthreads();

  // this lane's elements of a strip: rows row0 + 8 s + g, columns 8 j + 2 t + h
  Strips<SPW, TN, T1> p;
  Strips<SPW, TN, c128> v;
  product(p, P1, T, M, row0, g, t);
  __syncthreads();
#pragma unroll
  for (int s = 0; s < SPW; ++s) {
    const int r = row0 + 8 * s + g;
    if (r < M)
#pragma unroll
      for (int j = 0; j < TN; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c = 8 * j + 2 * t + h;
          const c128 x = cmk(p.cr[s][j][h], p.ci[s][j][h]);
          T[r * PT + c] = x;
          R[r * 8 * TN + c] = x;
        }
  }
  __syncthreads();
  for (int n = 1; n <= order; ++n) {
    const double a = 1.0 / double(n);
    if constexpr (KV > 0) {
      v.clear();
#pragma unroll
      for (int q = 0; q < KV; ++q)
        if (4 * q < M) v.step(fv[q], T, 4 * q + t, g);
    } else {
      product(v, Vw, T, M, row0, g, t);
    }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < SPW; ++s) {
      const int r = row0 + 8 * s + g;
      if (r < M)
#pragma unroll
        for (int j = 0; j < TN; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int c = 8 * j + 2 * t + h;
            const c128 x = cmul(cmk(0.0, a), cmk(v.cr[s][j][h], v.ci[s][j][h]));
            const c128 sum = cadd(R[r * 8 * TN + c], x);
            R[r * 8 * TN + c] = sum;
            T[r * PT + c] = n == order ? sum : x;  // the last product reads the sum
          }
    }
    __syncthreads();
  }
  product(p, P1, T, M, row0, g, t);
#pragma unroll
  for (int s = 0; s < SPW; ++s) {
    const int r = row0 + 8 * s + g;
    if (r < M)
#pragma unroll
      for (int j = 0; j < TN; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c = 8 * j + 2 * t + h;
          if (c < N) Sw[long(r) * N + c] = cmk(p.cr[s][j][h], p.ci[s][j][h]);
        }
  }
}

size_t smem_bytes(int M, int TN) {
  return (size_t((M + 3) / 4 * 4) * t_pitch(TN) + size_t(M) * 8 * TN) * sizeof(c128);
}

template <int SPW, int TN, int KV>
int run(cudaStream_t s, const void* P1, bool p1_real, const c128* V, long strideV, c128* S, long ldS,
        int W, int M, int N, int order) {
  const size_t smem = smem_bytes(M, TN);
  const int threads = 32 * ceil_div(M, 8 * SPW);
  auto go = [&](auto kern) -> int {
    AFQMC_TRY(allow_smem(kern, smem, smem_bytes(SPW == 2 ? 128 : KV > 0 ? 32 : 64, TN)));
    kern<<<W, threads, smem, s>>>(P1, V, strideV, S, ldS, M, N, order);
    return launch_status("taylor_c128_kernel");
  };
  return p1_real ? go(taylor_c128_kernel<SPW, TN, KV, true>)
                 : go(taylor_c128_kernel<SPW, TN, KV, false>);
}

template <int SPW, int KV>
int run_tn(cudaStream_t s, const void* P1, bool p1_real, const c128* V, long strideV, c128* S,
           long ldS, int W, int M, int N, int order) {
  switch ((N + 7) / 8) {
    case 1: return run<SPW, 1, KV>(s, P1, p1_real, V, strideV, S, ldS, W, M, N, order);
    case 2: return run<SPW, 2, KV>(s, P1, p1_real, V, strideV, S, ldS, W, M, N, order);
    case 3: return run<SPW, 3, KV>(s, P1, p1_real, V, strideV, S, ldS, W, M, N, order);
    default: return run<SPW, 4, KV>(s, P1, p1_real, V, strideV, S, ldS, W, M, N, order);
  }
}

}  // namespace

// M <= 64 (a strip per warp, two CTAs an SM where the accumulators are small): always.  Above that
// one CTA fits an SM by its registers and takes about the same time whatever the number of walkers, so
// with wide accumulators (N > 16) it depends on how many SMs the last wave leaves idle.  GEMM launches
// over this form, times of order 6 (1 to 1024 walkers; fill = W / 148 over the waves):
//   M = 48 to 64: 1.2 to 3.1 at every N from 32 walkers on
//   N <= 16, M = 65 to 128: 0.9 to 2.7 from 32 walkers on
//   N = 17..24: 0.86 to 1.15 at 32 walkers (fill 0.22), 1.2 at 60, 0.92 to 1.6 from 140 on
//   N = 25..32: M = 80 and 96: 0.77 at 149 walkers (0.50) and 300 (0.68), 0.83 at 445 (0.75), 0.84 to
//     0.89 at 600 (0.81), 1.03 at 256 (0.86), 1.12 at 296 (1.0), 0.92 to 0.95 at 1024 (0.99);
//     M = 100 to 128: 0.95 at 149, 0.97 to 1.02 at 200 (0.68) and 300, 1.27 at 296, 1.13 at 1024
bool taylor_c128_fits(int W, int M, int N) {
  if (N < 1 || N > 32 || M < 1 || M > 128 || smem_bytes(M, (N + 7) / 8) > 227 * 1024) return false;
  if (M <= 64 || N <= 16) return true;
  const double fill = double(W) / (double(NUM_SMS) * ceil_div(W, NUM_SMS));
  return fill >= (N <= 24 ? 0.3 : M <= 96 ? 0.85 : 0.65);
}

int taylor_c128(cudaStream_t s, const void* P1, bool p1_real, const c128* V, long strideV, c128* S,
                long ldS, int W, int M, int N, int order) {
  if (M <= 32) return run_tn<1, 8>(s, P1, p1_real, V, strideV, S, ldS, W, M, N, order);
  if (M <= 64) return run_tn<1, 0>(s, P1, p1_real, V, strideV, S, ldS, W, M, N, order);
  return run_tn<2, 0>(s, P1, p1_real, V, strideV, S, ldS, W, M, N, order);
}

}  // namespace afqmc
