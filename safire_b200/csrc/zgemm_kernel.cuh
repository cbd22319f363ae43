// The DMMA GEMM kernel behind zgemm.cuh: mma.sync m8n8k4 f64 on shared-memory tiles that arrive
// by cp.async.
//
// A CTA has nw warps (1..8, chosen per launch) and computes BM x BN = 8 nw x 8 TN outputs; each
// warp owns one 8-row strip of all BN columns.  One DMMA holds the SM's FP64 tensor path for about
// 4 cycles whatever the tile, and one A and TN B fragment loads feed TN (real x real) to 4 TN
// (complex x complex) of them, so the FP64 rate bounds every shape that fills its tiles.  What is
// lost is lost to padding: the tile is therefore fitted to the problem in steps of 8 in both
// directions (shape in zgemm.cu) instead of being 64 x 64.
//
// K runs in tiles of 16 through a ring of three shared-memory stages, one barrier per tile; the
// row pitches are padded so that the fragment loads are free of bank conflicts for 16-byte
// (complex) and 8-byte (real) elements.  With few output tiles, a cluster of `split` CTAs along z
// shares one tile's K range and adds the partial sums through distributed shared memory in rank
// order.
//
// Rates at 1024 walkers, of 35.5 TFLOP/s (cuBLAS DGEMM): 28.8 for the vHS pairs (K = 1600), 26.6
// for vbias (K = 10000; 400 tiles on 148 SMs leave a tenth idle), 24.2 for the Taylor product
// (200 x 50 x 200, padded to 224 x 56).  With 64 x 64 tiles throughout, and register staging in
// place of cp.async, the last ran at 16.
#pragma once

#include <cooperative_groups.h>

#include "dmma.cuh"
#include "zgemm.cuh"

namespace afqmc {
namespace zg {

constexpr int MAX_WARPS = 8;

// one element from global to shared memory, zero when `in` is false (the address is not read)
__device__ __forceinline__ void copy_async(c128* dst, const c128* src, bool in) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  const int bytes = in ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void copy_async(double* dst, const double* src, bool in) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  const int bytes = in ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

template <bool REAL>
struct Elem {
  using T = c128;
};
template <>
struct Elem<true> {
  using T = double;
};

// operand combination of an instantiation: transposed / conjugated / real A and B
template <bool AT_, bool AC_, bool AR_, bool BT_, bool BC_, bool BR_>
struct Op {
  static constexpr bool AT = AT_, AC = AC_, AR = AR_, BT = BT_, BC = BC_, BR = BR_;
  using TA = typename Elem<AR>::T;
  using TB = typename Elem<BR>::T;
  // pad (elements) of a stage's contiguous dimension: k-contiguous tiles pitch 20, m- or
  // n-contiguous ones 2 (complex) / 4 (real) past a multiple of 8
  static constexpr int PA = (AT && !AR) ? 2 : 4;
  static constexpr int PB = (!BT && !BR) ? 2 : 4;
  __host__ __device__ static constexpr int a_elems(int bm) {
    return AT ? BK * (bm + PA) : bm * (BK + PA);
  }
  __host__ __device__ static constexpr int b_elems(int bn) {
    return BT ? bn * (BK + PB) : BK * (bn + PB);
  }
  // a multiple of 16 bytes: bm, bn are multiples of 8
  __host__ __device__ static constexpr int stage_bytes(int bm, int bn) {
    return a_elems(bm) * int(sizeof(TA)) + b_elems(bn) * int(sizeof(TB));
  }
};

// SYM: B^T's rows are the (i, k) pairs of an M x M matrix whose row (i, k) equals row (k, i)
// (p.sym_m = M); a column tile is an 8 x 8 block of pairs with block(i) <= block(k), and each
// value goes to C[row][i M + k] and C[row][k M + i].
template <int TN, class O, bool SYM>
__global__ void __launch_bounds__(32 * MAX_WARPS, 2) zgemm_kernel(GemmParams p, int split) {
  using TA = typename O::TA;
  using TB = typename O::TB;
  constexpr int BN = 8 * TN;
  extern __shared__ __align__(16) unsigned char smem_raw[];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int NT = blockDim.x, BM = NT >> 2;
  const int g = lane >> 2, t = lane & 3;
  const int a_pitch = O::AT ? BM + O::PA : BK + O::PA;
  constexpr int b_pitch = O::BT ? BK + O::PB : BN + O::PB;
  const int a_bytes = O::a_elems(BM) * int(sizeof(TA));
  const int stage = a_bytes + O::b_elems(BN) * int(sizeof(TB));

  const long b = split > 1 ? 0 : blockIdx.z;
  const int rank = split > 1 ? blockIdx.z : 0;
  const int m0 = blockIdx.y * BM;
  int n0 = 0, sym_i0 = 0, sym_k0 = 0;
  if constexpr (SYM) {
    // upper-triangular block index -> (i block, k block)
    const int nb = (p.sym_m + 7) / 8;
    int r = blockIdx.x, ib = 0;
    while (r >= nb - ib) r -= nb - ib++;
    sym_i0 = 8 * ib;
    sym_k0 = 8 * (ib + r);
  } else {
    n0 = blockIdx.x * BN;
  }
  const TA* Ag = reinterpret_cast<const TA*>(p.A) + b * p.strideA;
  const TB* Bg = reinterpret_cast<const TB*>(p.B) + b * p.strideB;

  // this CTA's K tiles
  const int ktiles = (p.k + BK - 1) / BK;
  const int kt0 = int(long(ktiles) * rank / split), kt1 = int(long(ktiles) * (rank + 1) / split);

  // A copies: four elements per thread and stage
  const int a_row = O::AT ? tid / BM : tid >> 4;
  const int a_col = O::AT ? tid - a_row * BM : tid & 15;
  auto load_stage = [&](int kt) {
    unsigned char* st = smem_raw + ((kt - kt0) % STAGES) * stage;
    TA* as = reinterpret_cast<TA*>(st);
    TB* bs = reinterpret_cast<TB*>(st + a_bytes);
    const int k0 = kt * BK;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if constexpr (O::AT) {
        const int kk = a_row + 4 * i;
        const bool in = (m0 + a_col < p.m) && (k0 + kk < p.k);
        copy_async(as + kk * a_pitch + a_col,
                   in ? Ag + long(k0 + kk) * p.lda + (m0 + a_col) : Ag, in);
      } else {
        const int mm = a_row + (NT >> 4) * i;
        const bool in = (m0 + mm < p.m) && (k0 + a_col < p.k);
        copy_async(as + mm * a_pitch + a_col, in ? Ag + long(m0 + mm) * p.lda + (k0 + a_col) : Ag,
                   in);
      }
    }
    for (int e = tid; e < BN * BK; e += NT) {
      if constexpr (O::BT) {
        const int nn = e >> 4, kk = e & 15;
        bool in = k0 + kk < p.k;
        long row;
        if constexpr (SYM) {
          const int i = sym_i0 + (nn >> 3), k = sym_k0 + (nn & 7);
          in = in && i < p.sym_m && k < p.sym_m;
          row = long(i) * p.sym_m + k;
        } else {
          in = in && n0 + nn < p.n;
          row = n0 + nn;
        }
        copy_async(bs + nn * b_pitch + kk, in ? Bg + row * p.ldb + (k0 + kk) : Bg, in);
      } else {
        const int kk = e / BN, nn = e - kk * BN;
        const bool in = (n0 + nn < p.n) && (k0 + kk < p.k);
        copy_async(bs + kk * b_pitch + nn, in ? Bg + long(k0 + kk) * p.ldb + (n0 + nn) : Bg, in);
      }
    }
  };

  double accr[TN][2], acci[TN][2];
#pragma unroll
  for (int j = 0; j < TN; ++j) accr[j][0] = accr[j][1] = acci[j][0] = acci[j][1] = 0.0;

#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (kt0 + s < kt1) load_stage(kt0 + s);
    copy_commit();
  }
  for (int kt = kt0; kt < kt1; ++kt) {
    copy_wait<STAGES - 2>();
    __syncthreads();  // tile kt is here; every warp is done with the stage refilled next
    if (kt + STAGES - 1 < kt1) load_stage(kt + STAGES - 1);
    copy_commit();
    const unsigned char* st = smem_raw + ((kt - kt0) % STAGES) * stage;
    const TA* as = reinterpret_cast<const TA*>(st);
    const TB* bs = reinterpret_cast<const TB*>(st + a_bytes);
    const int krem = p.k - kt * BK;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 4) {
      if (kk >= krem) break;  // zeros past K
      const int r = warp * 8 + g, c = kk + t;
      TA fa = O::AT ? as[c * a_pitch + r] : as[r * a_pitch + c];
      if constexpr (O::AC) fa.y = -fa.y;
      TB fb[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const int cn = j * 8 + g;
        fb[j] = O::BT ? bs[cn * b_pitch + c] : bs[c * b_pitch + cn];
        if constexpr (O::BC) fb[j].y = -fb[j].y;
      }
      if constexpr (O::AR && O::BR) {
#pragma unroll
        for (int j = 0; j < TN; ++j) dmma(accr[j][0], accr[j][1], fa, fb[j]);
      } else if constexpr (O::AR) {
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          dmma(accr[j][0], accr[j][1], fa, fb[j].x);
          dmma(acci[j][0], acci[j][1], fa, fb[j].y);
        }
      } else if constexpr (O::BR) {
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          dmma(accr[j][0], accr[j][1], fa.x, fb[j]);
          dmma(acci[j][0], acci[j][1], fa.y, fb[j]);
        }
      } else {
        const double nai = -fa.y;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          dmma(accr[j][0], accr[j][1], fa.x, fb[j].x);
          dmma(acci[j][0], acci[j][1], fa.x, fb[j].y);
        }
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          dmma(accr[j][0], accr[j][1], nai, fb[j].y);
          dmma(acci[j][0], acci[j][1], fa.y, fb[j].x);
        }
      }
    }
  }

  c128* Cg = p.C + b * p.strideC;
  c128* Dg = p.D ? p.D + b * p.strideD : nullptr;
  const bool use_beta = (p.beta.x != 0.0 || p.beta.y != 0.0);
  auto store = [&](int row, int cl, c128 acc) {  // row of C, column of this tile
    if (row >= p.m) return;
    c128 v = cmul(p.alpha, acc);
    if constexpr (SYM) {
      const int i = sym_i0 + (cl >> 3), k = sym_k0 + (cl & 7);
      if (i >= p.sym_m || k >= p.sym_m) return;
      c128* Cr = Cg + long(row) * p.ldc;
      Cr[long(i) * p.sym_m + k] = v;
      if (sym_i0 != sym_k0) Cr[long(k) * p.sym_m + i] = v;
    } else {
      const int col = n0 + cl;
      if (col >= p.n) return;
      const long oc = long(row) * p.ldc + col;
      if (use_beta) v = cadd(v, cmul(p.beta, Cg[oc]));
      Cg[oc] = v;
      if (Dg) {
        const long od = long(row) * p.ldd + col;
        Dg[od] = p.d_store ? v : cadd(Dg[od], v);
      }
    }
  };

  if (split > 1) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    c128* red = reinterpret_cast<c128*>(smem_raw);
    copy_wait<0>();
    __syncthreads();
#pragma unroll
    for (int j = 0; j < TN; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        red[(warp * 8 + g) * BN + j * 8 + 2 * t + h] = cmk(accr[j][h], acci[j][h]);
    cl.sync();
    // the cluster's CTAs take the tile's elements in turn
    for (int e = rank * NT + tid; e < BM * BN; e += split * NT) {
      c128 acc = cmk(0.0, 0.0);
      for (int r = 0; r < split; ++r) acc = cadd(acc, cl.map_shared_rank(red, r)[e]);
      store(m0 + e / BN, e % BN, acc);
    }
    cl.sync();  // no CTA leaves while its partial sums are being read
    return;
  }
#pragma unroll
  for (int j = 0; j < TN; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      store(m0 + warp * 8 + g, j * 8 + 2 * t + h, cmk(accr[j][h], acci[j][h]));
}

template <int TN, class O, bool SYM>
int launch(cudaStream_t s, int batch, const GemmParams& p, const Shape& sh) {
  auto kern = zgemm_kernel<TN, O, SYM>;
  constexpr int bn = 8 * TN;
  const int bm = 8 * sh.warps;
  size_t smem = size_t(STAGES) * O::stage_bytes(bm, bn);
  if (sh.split > 1 && smem < size_t(bm) * bn * sizeof(c128)) smem = size_t(bm) * bn * sizeof(c128);
  constexpr size_t ring = STAGES * size_t(O::stage_bytes(8 * MAX_WARPS, bn));
  constexpr size_t sums = size_t(8 * MAX_WARPS) * bn * sizeof(c128);
  AFQMC_TRY(allow_smem(kern, smem, ring > sums ? ring : sums));  // of any shape
  unsigned gx = ceil_div(p.n, bn);
  if (SYM) {
    const unsigned nb = ceil_div(p.sym_m, 8);
    gx = nb * (nb + 1) / 2;
  }
  const dim3 grid(gx, ceil_div(p.m, bm), sh.split > 1 ? sh.split : batch);
  if (sh.split > 1) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(32 * sh.warps);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 1;
    at.val.clusterDim.y = 1;
    at.val.clusterDim.z = unsigned(sh.split);
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    AFQMC_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, p, sh.split));
  } else {
    kern<<<grid, 32 * sh.warps, smem, s>>>(p, 1);
  }
  return launch_status("zgemm_kernel");
}

template <class O>
int launch_tn(cudaStream_t s, int batch, const GemmParams& p, const Shape& sh) {
  switch (sh.tn) {
    case 1: return launch<1, O, false>(s, batch, p, sh);
    case 2: return launch<2, O, false>(s, batch, p, sh);
    case 3: return launch<3, O, false>(s, batch, p, sh);
    case 4: return launch<4, O, false>(s, batch, p, sh);
    case 5: return launch<5, O, false>(s, batch, p, sh);
    case 6: return launch<6, O, false>(s, batch, p, sh);
    case 7: return launch<7, O, false>(s, batch, p, sh);
    default: return launch<8, O, false>(s, batch, p, sh);
  }
}

}  // namespace zg
}  // namespace afqmc
