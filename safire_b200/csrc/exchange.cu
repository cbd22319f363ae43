// Fused exchange / Coulomb contraction of the local energy on the tensor cores.
//
// Reference: Real3IndexFactorization::energy_impl (src/AFQMC/HamiltonianOperations/
// Real3IndexFactorization.hpp:476-590) forms T[w,b,n,a] = sum_k G[w,b,k] Lnak[n,a,k] in chunks of
// Cholesky vectors (71 GB at M=200, N=50, Nc=1600, W=1024 if materialised) and reduces
// EXX[w] += -scl/2 sum_{n,a,b} T[w,a,n,b] T[w,b,n,a] and Kl[w,n] = sum_a T[w,a,n,a].
// Here T never leaves the SM: a persistent kernel walks tiles of NV Cholesky vectors x NW walkers;
// each tile is one 128 x 2 NW SB tcgen05 accumulator (split products, FP32 in TMEM):
//   rows   = NV slots of SA (a = 0..N-1, the rest zero)       <- TMA box {128 bytes, SA, NV} of Lnak
//   cols   = real parts, then imaginary parts of NW slots of SB (b = 0..N-1)
//                                                             <- TMA boxes {128 bytes, SB, NW} of G
// so one MMA multiplies a vector plane with both parts of the walkers: an accumulator row is
// a column of T_n, and the transposed pairing T[a][b] T[b][a] does not mind.  The epilogue warps
// stage the lower triangle of each N x N block in shared memory, form the sum over pairs a < b
// and the diagonal per (walker, n), in FP64 from the partial sums on, and store them; the next
// tile's MMAs run meanwhile into the second TMEM accumulator.
//
// What bounds it is the MMA path together with the operands' way from L2 (85 KB per 64 orbitals for
// 1248 cycles of MMA at N = 50).  With the walkers as the 128 rows and the (real) vectors as the
// columns, each part of G met each vector plane in an MMA of its own, 112 columns wide: 45.6 KB of
// shared-memory operands per 16-element K step at N = 50, against 31.5 KB here for the same
// products; 15.6 ms against 14.7 ms for 1024 walkers, 1600 vectors, M = 200 (14.1 ms of the old form
// without its epilogue's work).  CTA pairs (cta_group::2, half of B each) took 18.1 ms.
// Slots fitted to N (64-row slots for every N before) let a tile hold four times the pairs at N = 25.
#include <cudaTypedefs.h>

#include "energy.cuh"
#include "mixed.cuh"
#include "tc.cuh"

namespace afqmc {
namespace {

constexpr int XT_THREADS = 192;  // warp 0 TMA, warp 1 MMA, warps 2-5 epilogue
constexpr int XBK = 32;
constexpr int X_ROWS = 128;
constexpr int X_ACC = 256;       // TMEM columns per accumulator (two of them)
constexpr int X_STRIP = 12;      // walker groups per strip of the tile order
constexpr int NBLK_DEFAULT = 64; // vector pairs per L2 block of the tile order (autotuned: 16..128)
constexpr size_t X_SMEM_MAX = 232448;

struct XParams {
  CUtensorMap a[2];  // Lnak planes as {M, N, Nc}: hi, lo (real trial)
  CUtensorMap b[4];  // G planes as {M, N, W}: re_hi, re_lo, im_hi, im_lo (1 product: re_hi, im_hi)
  int W, N, Nc, M;
  int NV;            // vectors per tile (128 / SA)
  int NW, SB;        // walkers per tile and their column slot; NW SB a multiple of 8, at most 128
  int stages, stg_bytes;
  c128* exx;         // [W][Nc] += sum_{a,b} T[b][a] T[a][b]
  c128* kl;          // [W][Nc] += trace T
  const float* ginv; // FP16 operands: per-walker inverse scale of G (null for TF32)
  float linv;        // FP16 operands: inverse scale of Lnak
  int nblk;          // vector groups per L2 block of the tile order
  unsigned* err;
};

__device__ __forceinline__ void named_bar(int id, int n) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                 "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// tile t -> (walker group, vector group): blocks of nblk vector groups, whose Lnak planes stay in
// L2 while every walker passes; inside a block, strips of X_STRIP walker groups with the walker
// group fastest, so that the tiles in flight at a time share both their operands (about
// 12 x 12 groups on 148 SMs)
__device__ __forceinline__ void tile_coords(long t, int WP, int NP, int nblk, int& wp, int& np) {
  const long per_blk = long(WP) * nblk;
  const int nb = int(t / per_blk);
  const int width = min(nblk, NP - nb * nblk);
  const long within = t - nb * per_blk, per_strip = long(X_STRIP) * width;
  const int strip = int(within / per_strip);
  const int rows = min(X_STRIP, WP - strip * X_STRIP);
  const int r = int(within - strip * per_strip);
  wp = strip * X_STRIP + r % rows;
  np = nb * nblk + r / rows;
}

// Sums of v[0..3] over groups of G lanes (16 or 32): the lanes whose bits (G/2, G/4) are q hold
// the sum of v[q].  Each step halves what a lane carries, six double shuffles in place of twenty.
template <int G>
__device__ __forceinline__ double reduce4(const double (&v)[4], int lane) {
  const bool h1 = lane & (G / 2), h2 = lane & (G / 4);
  double a = h1 ? v[2] : v[0], b = h1 ? v[3] : v[1];
  a += __shfl_xor_sync(0xffffffffu, h1 ? v[0] : v[2], G / 2);
  b += __shfl_xor_sync(0xffffffffu, h1 ? v[1] : v[3], G / 2);
  double x = h2 ? b : a;
  x += __shfl_xor_sync(0xffffffffu, h2 ? a : b, G / 4);
#pragma unroll
  for (int o = G / 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// SA: rows per vector slot (16, 32, 64 >= N)
template <int SA, int NSPLIT, bool F16>
__global__ void __launch_bounds__(XT_THREADS, 1) exchange_tc_kernel(const __grid_constant__ XParams p) {
  // 128 bytes of K per stage and operand row: 32 TF32 or 64 FP16 elements; 32 bytes per MMA
  constexpr int XBKE = F16 ? 2 * XBK : XBK;
  constexpr int KSTEP = F16 ? 16 : 8;
  constexpr int NA = NSPLIT == 3 ? 2 : 1;      // planes of each part
  constexpr int NCOL = SA == 64 ? 56 : SA;     // accumulator columns a thread holds per walker
  constexpr int A_TILE = X_ROWS * XBK * 4;
  // The pairs a < b once, or all of them: half the lanes' accesses to shared memory against a
  // comparison of each lane's a with every b.  Measured (M = 104, N = 40, 400 vectors, 1024 walkers),
  // the triangle and all pairs: FP16 3.01 and 3.22 ms, TF32 3.55 and 3.15.
  constexpr bool ALL_PAIRS = !F16;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int ncols = p.NW * p.SB;               // columns of one part
  const int part = ncols * XBK * 4;            // bytes of one part of a B plane
  const int stage = NA * (A_TILE + 2 * part);
  const int STAGES = p.stages;
  float2* st2 = reinterpret_cast<float2*>(base + size_t(STAGES) * stage);  // [NV][N][PITCH]
  uint64_t* full = reinterpret_cast<uint64_t*>(base + size_t(STAGES) * stage + p.stg_bytes);
  uint64_t* empty = full + 4;
  uint64_t* acc_full = empty + 4;          // [2]
  uint64_t* acc_empty = acc_full + 2;      // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  double* red = reinterpret_cast<double*>(tmem_slot + 4);  // [4 lane quarters][4] partial sums
  int* const agree = reinterpret_cast<int*>(red + 16);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int WP = (p.W + p.NW - 1) / p.NW, NP = (p.Nc + p.NV - 1) / p.NV;
  const long ntiles = long(WP) * NP;
  const int N = p.N;
  const int PITCH = N | 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&acc_full[b], 1);
      tc::mbar_init(&acc_empty[b], 128);
    }
    *abort_flag = 0;
    tc::fence_mbar_init();
    for (int q = 0; q < NA; ++q) tc::prefetch_tmap(&p.a[q]);
    for (int q = 0; q < 2 * NA; ++q) tc::prefetch_tmap(&p.b[q]);
  }
  if (warp == 1) {
    tc::tmem_alloc(tmem_slot, 512);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t taddr = *tmem_slot;
  const int nk = (p.M + XBKE - 1) / XBKE;

  if (warp == 0) {
    if (lane == 0) {
      int s = 0;              // stage ring position and the parity of its last release
      unsigned par = 1;       // the first pass over the ring finds every stage free
      for (long t = blockIdx.x; t < ntiles; t += gridDim.x) {
        int wp, np;
        tile_coords(t, WP, NP, p.nblk, wp, np);
        bool ok = true;
        for (int kc = 0; kc < nk; ++kc) {
          if (!tc::mbar_wait(&empty[s], par, p.err, abort_flag)) {
            ok = false;
            break;
          }
          unsigned char* st = base + size_t(s) * stage;
          tc::mbar_arrive_expect_tx(&full[s], unsigned(stage));
#pragma unroll
          for (int q = 0; q < NA; ++q)
            tc::tma_load_3d(st + q * A_TILE, &p.a[q], &full[s], kc * XBKE, 0, p.NV * np);
          // B plane q (hi, lo): real part, then imaginary part
#pragma unroll
          for (int q = 0; q < NA; ++q) {
            unsigned char* bs = st + NA * A_TILE + q * 2 * part;
            tc::tma_load_3d(bs, &p.b[q], &full[s], kc * XBKE, 0, p.NW * wp);
            tc::tma_load_3d(bs + part, &p.b[NA + q], &full[s], kc * XBKE, 0, p.NW * wp);
          }
          if (++s == STAGES) {
            s = 0;
            par ^= 1u;
          }
        }
        if (!ok) break;
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t ID = tc::idesc_split<F16>(X_ROWS, 2 * ncols, false);
      int s = 0;
      unsigned par = 0;
      long ti = 0;
      bool ok = true;
      for (long t = blockIdx.x; t < ntiles && ok; t += gridDim.x, ++ti) {
        const int buf = int(ti & 1);
        // wait for the epilogue to have drained this accumulator (tile ti-2)
        if (ti >= 2) {
          if (!tc::mbar_wait(&acc_empty[buf], unsigned((ti / 2) - 1) & 1u, p.err, abort_flag)) {
            ok = false;
            break;
          }
        }
        tc::tc_fence_after();
        const uint32_t d = taddr + uint32_t(buf * X_ACC);
        for (int kc = 0; kc < nk; ++kc) {
          if (!tc::mbar_wait(&full[s], par, p.err, abort_flag)) {
            ok = false;
            break;
          }
          tc::tc_fence_after();
          const uint32_t sa = tc::smem_u32(base + size_t(s) * stage);
          const uint32_t sb = sa + NA * A_TILE;
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            if (kc * XBKE + kk * KSTEP >= p.M) break;  // zero fill past K
            auto A = [&](int q) { return tc::sdesc_sw128(sa + q * A_TILE) + uint64_t(2 * kk); };
            auto B = [&](int q) { return tc::sdesc_sw128(sb + q * 2 * part) + uint64_t(2 * kk); };
            const uint32_t acc0 = (kc > 0 || kk > 0) ? 1u : 0u;
            // (Tr, Ti)^T = L (Gr, Gi)^T: hi*hi + lo*hi + hi*lo
            tc::mma_split<F16>(d, A(0), B(0), ID, acc0);
            if constexpr (NSPLIT == 3) {
              tc::mma_split<F16>(d, A(1), B(0), ID, 1);
              tc::mma_split<F16>(d, A(0), B(1), ID, 1);
            }
          }
          tc::mma_commit(&empty[s]);
          if (++s == STAGES) {
            s = 0;
            par ^= 1u;
          }
        }
        if (!ok) break;
        tc::mma_commit(&acc_full[buf]);
      }
    }
  } else {
    // epilogue: TMEM lane quarter q = warp % 4; lane L = row of the accumulator = (vector, a)
    const int q = warp & 3;
    const int L = q * 32 + lane;
    const int v = L / SA, a = L % SA;
    const int et = threadIdx.x - 64;  // 0..127
    // the thread that adds component ci (exx re, im, kl re, im) of vector vo to the output
    constexpr int G = SA >= 32 ? 32 : 16;
    const int ci = SA == 64 ? (et & 3) : (lane & (G / 2) ? 2 : 0) + (lane & (G / 4) ? 1 : 0);
    const int vo = SA == 64 ? (et >> 2) : v;
    const bool upd = SA == 64 ? et < 8 : (lane & (G / 4 - 1)) == 0;
    long ti = 0;
    for (long t = blockIdx.x; t < ntiles; t += gridDim.x, ++ti) {
      int wp, np;
      tile_coords(t, WP, NP, p.nblk, wp, np);
      const int buf = int(ti & 1);
      // the four epilogue warps meet at named barriers below: they leave the loop together, on
      // the outcome of all four waits (a wait that gave up on one warp ends every warp's loop)
      bool ok = tc::mbar_wait_warp(&acc_full[buf], unsigned(ti / 2) & 1u, p.err, abort_flag);
      if (lane == 0) agree[q] = ok ? 0 : 1;
      named_bar(1, 128);
      ok = (agree[0] | agree[1] | agree[2] | agree[3]) == 0;
      named_bar(1, 128);
      tc::tc_fence_after();
      if (!ok) break;
      const bool valid = a < N && np * p.NV + v < p.Nc;
      const uint32_t trow = taddr + (uint32_t(q * 32) << 16) + uint32_t(buf * X_ACC);
      const int nw = min(p.NW, p.W - wp * p.NW);
      const int no = np * p.NV + vo;
      float2* const row = st2 + (v * N + a) * PITCH;
      const float2* const col = st2 + v * N * PITCH + a;
#pragma unroll 1
      for (int wl = 0; wl < nw; ++wl) {
        const int w = wp * p.NW + wl;
        // row a of the block (columns b) into registers, and its lower triangle (or the whole row)
        // into the staging block, from which the rows above (or all) read it as their column
        float vr[NCOL], vi[NCOL];
        {
          const uint32_t cr = trow + uint32_t(wl * p.SB), ci_ = cr + uint32_t(ncols);
#pragma unroll
          for (int c = 0; c < NCOL; c += 8)
            if (c < N) {
              tmem_ld8(cr + c, vr + c);
              tmem_ld8(ci_ + c, vi + c);
            }
          tc::tmem_ld_wait();
        }
        if (wl == nw - 1) {
          tc::tc_fence_before();
          tc::mbar_arrive(&acc_empty[buf]);  // accumulator free for tile ti+2
        }
        if (valid) {
#pragma unroll
          for (int b = 0; b < NCOL; ++b)
            if (ALL_PAIRS ? b < N : b <= a) row[b] = make_float2(vr[b], vi[b]);
        }
        // the running sum this thread adds to, fetched now so its latency hides behind the loop
        double* out = nullptr;
        double old = 0.0;
        if (upd && no < p.Nc) {
          out = reinterpret_cast<double*>((ci & 2 ? p.kl : p.exx) + long(w) * p.Nc + no) + (ci & 1);
          old = *out;
        }
        named_bar(1, 128);
        // x = T[a][a]^2 + 2 sum_{b > a} T[a][b] T[b][a], or sum_b T[a][b] T[b][a] where the
        // block is whole;  tr = T[a][a].  The sum over b runs in FP32 with four independent accumulator pairs; the partial sums are widened to FP64 for
        // every later sum.
        double v4[4] = {0.0, 0.0, 0.0, 0.0};
        if (valid) {
          float xr[4] = {0.f, 0.f, 0.f, 0.f}, xi[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int b = 0; b < NCOL; ++b)
            if (b < N && (ALL_PAIRS || b > a)) {
              const float2 u = col[b * PITCH];  // T[b][a]
              xr[b & 3] = fmaf(vr[b], u.x, fmaf(-vi[b], u.y, xr[b & 3]));
              xi[b & 3] = fmaf(vr[b], u.y, fmaf(vi[b], u.x, xi[b & 3]));
            }
          const float2 d = row[a];
          const double dr = d.x, di = d.y;
          v4[0] = (double(xr[0]) + double(xr[1])) + (double(xr[2]) + double(xr[3]));
          v4[1] = (double(xi[0]) + double(xi[1])) + (double(xi[2]) + double(xi[3]));
          if (!ALL_PAIRS) {
            v4[0] = 2.0 * v4[0] + (dr * dr - di * di);
            v4[1] = 2.0 * v4[1] + 2.0 * dr * di;
          }
          v4[2] = dr;
          v4[3] = di;
        }
        double x = reduce4<G>(v4, lane);
        if constexpr (SA == 64) {
          if ((lane & 7) == 0) red[q * 4 + (lane >> 3)] = x;
        }
        // every thread is past its reads of the staging block (and red is complete): the block is
        // rewritten for the next walker after this barrier, red after the next one
        named_bar(1, 128);
        if (out) {
          if constexpr (SA == 64) x = red[(2 * vo) * 4 + ci] + red[(2 * vo + 1) * 4 + ci];
          // undo the power-of-two operand scales (exact)
          const double f = F16 ? double(p.ginv[w]) * double(p.linv) : 1.0;
          *out = old + x * (ci & 2 ? f : f * f);
        }
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 1) tc::tmem_dealloc(taddr, 512);
}

int g_num_sms = 0;

}  // namespace

int make_plane_map_3d_es(CUtensorMap* map, const void* base, int esize, long k, long rows,
                         long row_stride, long batch, long batch_stride, int box_rows,
                         int box_batch);

namespace {
template <int SA, int NSPLIT, bool F16>
int launch_exchange(cudaStream_t s, const XParams& p, int grid, size_t smem) {
  AFQMC_TRY(allow_smem(exchange_tc_kernel<SA, NSPLIT, F16>, smem, X_SMEM_MAX));
  exchange_tc_kernel<SA, NSPLIT, F16><<<grid, XT_THREADS, smem, s>>>(p);
  return launch_status("exchange_tc_kernel");
}
template <int SA>
int launch_exchange_sa(cudaStream_t s, const XParams& p, int grid, size_t smem, int nsplit,
                       bool f16) {
  if (nsplit == 3)
    return f16 ? launch_exchange<SA, 3, true>(s, p, grid, smem)
               : launch_exchange<SA, 3, false>(s, p, grid, smem);
  return f16 ? launch_exchange<SA, 1, true>(s, p, grid, smem)
             : launch_exchange<SA, 1, false>(s, p, grid, smem);
}
}  // namespace

// T-free exchange: exx[w][n] += sum_{a,b} T[b][a]T[a][b], kl[w][n] += trace T for spin block sp.
// G planes: [W][ldG] with the spin block at element offset `off` (rows of M); Lnak planes
// [Nc][N][M]; FP32 (esize 4, TF32 split) or FP16 (esize 2, FP16 split: G rows scaled per walker,
// g_inv[w] and l_inv the inverse scales).
int exchange_fused_tc(cudaStream_t s, const void* const Gp[4], int esize, long ldG, long off,
                      const void* const Lp[2], int W, int N, int Nc, int M, int nsplit,
                      const float* g_inv, float l_inv, c128* exx, c128* kl, unsigned* err,
                      int nblk) {
  if (N > 50 || N < 1) {
    set_error_detail("exchange_fused_tc: N = %d outside 1..50", N);
    return AFQMC_ERR_UNSUPPORTED;
  }
  const bool f16 = esize == 2;
  if (f16 && !g_inv) {
    set_error_detail("exchange_fused_tc: FP16 planes without their scales");
    return AFQMC_ERR_ARG;
  }
  const int SA = N <= 16 ? 16 : (N <= 32 ? 32 : 64);
  XParams p{};
  p.W = W;
  p.N = N;
  p.Nc = Nc;
  p.M = M;
  p.NV = X_ROWS / SA;
  // Walkers per tile: the columns of one part, NW slots of SB >= N, fill at most 128 (half an
  // accumulator) in multiples of 8; the most walkers per column wins, the wider tile on a tie.
  double best = 0.0;
  for (int nw = 1; nw <= 16; ++nw) {
    const int step = nw % 8 == 0 ? 1 : (nw % 4 == 0 ? 2 : (nw % 2 == 0 ? 4 : 8));
    const int sb = (N + step - 1) / step * step;
    if (nw * sb > 128) continue;
    // a tile's cost: its columns, and the 64 rows' worth of the vector planes it loads besides
    const double rate = double(nw) / (nw * sb + 64);
    if (rate > best) {
      best = rate;
      p.NW = nw;
      p.SB = sb;
    }
  }
  const int na = nsplit == 3 ? 2 : 1;
  for (int q = 0; q < na; ++q) {
    AFQMC_TRY(make_plane_map_3d_es(&p.a[q], Lp[q], esize, M, N, M, Nc, long(N) * M, SA, p.NV));
    // G's planes are re_hi, re_lo, im_hi, im_lo; the kernel's b: the hi (and lo) planes of the
    // real part, then those of the imaginary part
    for (int part = 0; part < 2; ++part)
      AFQMC_TRY(make_plane_map_3d_es(&p.b[part * na + q],
                                     static_cast<const char*>(Gp[2 * part + q]) + off * esize, esize,
                                     M, N, M, W, ldG, p.SB, p.NW));
  }
  p.exx = exx;
  p.kl = kl;
  p.ginv = g_inv;
  p.linv = l_inv;
  p.nblk = 2 * (nblk > 0 ? nblk : NBLK_DEFAULT) / p.NV;  // vector pairs -> vector groups
  if (p.nblk < 1) p.nblk = 1;
  p.err = err;
  const size_t stage = size_t(na) * (X_ROWS + 2 * p.NW * p.SB) * XBK * 4;
  p.stg_bytes = (p.NV * N * (N | 1) * 8 + 15) / 16 * 16;
  const size_t fixed = size_t(p.stg_bytes) + 1024 /*alignment*/ + 512 /*barriers, sums*/;
  p.stages = int((X_SMEM_MAX - fixed) / stage);
  if (p.stages > 4) p.stages = 4;
  const size_t smem = p.stages * stage + fixed;
  if (g_num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  const long ntiles = long(ceil_div(W, p.NW)) * ceil_div(Nc, p.NV);
  const int grid = int(ntiles < g_num_sms ? ntiles : g_num_sms);
  if (SA == 16) return launch_exchange_sa<16>(s, p, grid, smem, nsplit, f16);
  if (SA == 32) return launch_exchange_sa<32>(s, p, grid, smem, nsplit, f16);
  return launch_exchange_sa<64>(s, p, grid, smem, nsplit, f16);
}

}  // namespace afqmc
