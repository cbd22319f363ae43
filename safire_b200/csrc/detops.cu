// det_ops on the device: batched overlap matrices, LU log-determinants, inverses, mixed density
// matrices, Taylor propagation and QR re-orthonormalisation.
//
// Reference: src/AFQMC/SlaterDeterminantOperations/density_matrix.hpp (log_overlap_impl 113-156,
// MixedDensityMatrix 535-601, inverse_logdet 43-111), determinants_impl.hpp (log-det conventions),
// propagate.hpp (apply_expM 41-70, propagate_impl 238-298), orthogonalize.hpp (131-169).
#include "detops.cuh"
#include "dmma.cuh"
#include "zgemm.cuh"

namespace afqmc {

__device__ __forceinline__ c128 wrap_imag(c128 z) {
  const double pi = 3.14159265358979323846;
  double im = z.y;
  if (im > pi) {
    while (im > pi) im -= 2 * pi;
  } else if (im < -pi) {
    while (im < -pi) im += 2 * pi;
  }
  return cmk(z.x, im);
}

// log(d + DBL_MIN) or log(-1*d + DBL_MIN), as log_determinant_from_getrf_impl writes it
__device__ __forceinline__ c128 log_pivot(c128 d, bool swapped) {
  const double small = 2.2250738585072014e-308;
  c128 v = swapped ? cmul(cmk(-1.0, 0.0), d) : d;
  return clog(cmk(v.x + small, v.y + 0.0));
}

// ---------------------------------------------------------------------------------------------
// Gauss-Jordan elimination with partial pivoting (pivot = first max |re|+|im|, as izamax) on
// [A | I] in shared memory.  The pivots are the U diagonal of getrf with the same row
// interchanges, so the log-determinant follows log_determinant_from_getrf; the right half ends as
// A^{-1} (zero for a singular A, as getri_or_zero).  Without the inverse only the trailing
// submatrix is eliminated (plain LU) and the matrix needs a quarter of the shared memory, so more
// matrices share an SM.  One CTA per matrix, 8 warps: warp 0 finds the pivot, the pivot row, the
// old row k and the scaled multipliers are snapshotted, then every thread updates its
// (rows ty+8r) x (cols k+1+tx+32c) elements from the snapshots only: three barriers per step and
// no element read after another thread wrote it in the same phase.
// ---------------------------------------------------------------------------------------------
constexpr int GJ_THREADS = 256;
constexpr size_t GJ_SMEM_MAX = 227 * 1024 - 64;  // an SM's shared memory less the statics

template <bool INVERT>
__global__ void __launch_bounds__(GJ_THREADS) gj_logdet_kernel(const c128* __restrict__ A,
                                                                long strideA,
                                                                c128* __restrict__ Ainv,
                                                                long strideInv,
                                                                c128* __restrict__ ovlp, int N,
                                                                c128 post_scale, c128 post_add) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int P = INVERT ? 2 * N : N;  // columns of the augmented matrix
  const int PP = P | 1;              // odd pitch: conflict-free column walks
  c128* a = reinterpret_cast<c128*>(smem_raw);  // [N][PP]
  c128* rbuf = a + size_t(N) * PP;              // pivot row (post-swap row k) [P]
  c128* kbuf = rbuf + P;                        // old row k [P]
  c128* mbuf = kbuf + P;                        // scaled multipliers of the post-swap rows [N]
  c128* piv_val = mbuf + N;                     // [N]
  int* piv_swapped = reinterpret_cast<int*>(piv_val + N);
  __shared__ int s_piv;
  __shared__ int s_singular;
  __shared__ c128 s_dinv;

  const long w = blockIdx.x;
  const c128* Aw = A + w * strideA;
  const int tid = threadIdx.x;
  const int tx = tid & 31, ty = tid >> 5;
  for (int i = ty; i < N; i += GJ_THREADS / 32) {
    for (int j = tx; j < N; j += 32) a[i * PP + j] = Aw[long(i) * N + j];
    if (INVERT)
      for (int j = tx; j < N; j += 32) a[i * PP + N + j] = cmk(i == j ? 1.0 : 0.0, 0.0);
  }
  if (tid == 0) s_singular = 0;
  __syncthreads();

  for (int k = 0; k < N; ++k) {
    // 1. pivot search in column k, rows k..N-1 (warp 0)
    if (ty == 0) {
      double best = -1.0;
      int bi = N;
      for (int i = k + tx; i < N; i += 32) {
        const double v = cabs1(a[i * PP + k]);
        if (v > best) {
          best = v;
          bi = i;
        }
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, best, off);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
        if (ov > best || (ov == best && oi < bi)) {
          best = ov;
          bi = oi;
        }
      }
      if (tx == 0) {
        if (bi >= N) bi = k;  // a column of NaNs: zero pivot at row k
        s_piv = bi;
        piv_swapped[k] = (bi != k);
        const c128 d = a[bi * PP + k];
        piv_val[k] = d;
        if (!(best > 0.0)) {
          s_singular = 1;
          s_dinv = cmk(0, 0);
        } else {
          s_dinv = cdiv(cmk(1.0, 0.0), d);
        }
      }
    }
    __syncthreads();
    const int p = s_piv;
    const c128 dinv = s_dinv;
    const bool zero = (dinv.x == 0.0 && dinv.y == 0.0);
    // 2. snapshots: pivot row, old row k, multipliers (column k of the post-swap rows) * dinv
    for (int j = k + tid; j < P; j += GJ_THREADS) {
      rbuf[j] = a[p * PP + j];
      kbuf[j] = a[k * PP + j];
    }
    for (int i = (INVERT ? 0 : k) + tid; i < N; i += GJ_THREADS) {
      const c128 c = (i == k) ? a[p * PP + k] : ((i == p) ? a[k * PP + k] : a[i * PP + k]);
      mbuf[i] = cmul(c, dinv);
    }
    __syncthreads();
    // 3. row swap + elimination (+ pivot-row scaling for the inverse)
    const int r0 = INVERT ? 0 : k;
    for (int i = r0 + ty; i < N; i += GJ_THREADS / 32) {
      if (i == k) {
        for (int j = k + 1 + tx; j < P; j += 32)
          a[k * PP + j] = (INVERT && !zero) ? cmul(rbuf[j], dinv) : rbuf[j];
      } else {
        const c128 m = mbuf[i];
        const bool from_k = (i == p);
        for (int j = k + 1 + tx; j < P; j += 32) {
          const c128 src = from_k ? kbuf[j] : a[i * PP + j];
          a[i * PP + j] = zero ? src : csub(src, cmul(m, rbuf[j]));
        }
      }
    }
    __syncthreads();
  }

  // log det: sum_k log(+-U_kk + DBL_MIN), accumulated onto ovlp, imaginary part wrapped
  if (ty == 0) {
    double sr = 0.0, si = 0.0;
    for (int k = tx; k < N; k += 32) {
      const c128 l = log_pivot(piv_val[k], piv_swapped[k] != 0);
      sr += l.x;
      si += l.y;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      sr += __shfl_xor_sync(0xffffffffu, sr, off);
      si += __shfl_xor_sync(0xffffffffu, si, off);
    }
    if (tx == 0) {
      c128 res = cadd(ovlp[w], cmk(sr, si));
      res = wrap_imag(res);
      ovlp[w] = cadd(cmul(post_scale, res), post_add);
    }
  }
  if (INVERT) {
    c128* Iw = Ainv + w * strideInv;
    const bool sing = s_singular != 0;
    for (int i = ty; i < N; i += GJ_THREADS / 32)
      for (int j = tx; j < N; j += 32) Iw[long(i) * N + j] = sing ? cmk(0.0, 0.0) : a[i * PP + N + j];
  }
}

// ---------------------------------------------------------------------------------------------
// Warp-resident Gauss-Jordan / LU for N <= 16: G lanes (the power of two >= N) hold one matrix, a
// row per lane and its columns in registers, 32 / G matrices to a warp, no block barriers.
// Partial pivoting as izamax; the pivots give the log determinant, the in-place Gauss-Jordan the
// inverse.  Row interchanges move no data: each lane knows the logical index of its row.  The
// columns are kept rotated so that the pivot column of every step is register 0 (the update of column
// j writes register j - 1, and the finished column goes to register NC - 1), so the step loop is not
// unrolled over k and no register index depends on N; the NC - N registers past the matrix rotate
// along as zeros that nothing reads.  The pivot row reaches the other lanes by shuffles (G <= 8) or
// through a shared-memory row.
// What bounds it is the latency of the N dependent steps; small matrices are many (a trial of 34
// determinants inverts 52224 of 3 x 3 per spin and step), so the point is matrices in flight: a
// 128-thread CTA per matrix took 232 us for those, this form 10.4.
// ---------------------------------------------------------------------------------------------
constexpr int GW_WARPS = 4;

template <int G, int NC, bool INVERT>
__global__ void __launch_bounds__(32 * GW_WARPS)
    gj_warp_kernel(const c128* __restrict__ A, long strideA, c128* Ainv, long strideInv,
                   c128* __restrict__ ovlp, int W, int N, c128 post_scale, c128 post_add) {
  static_assert(NC <= G, "a row per lane");
  constexpr unsigned FULL = 0xffffffffu;
  constexpr bool SMEM_ROW = G > 8;
  __shared__ c128 rows[SMEM_ROW ? GW_WARPS : 1][2][SMEM_ROW ? 32 : 1];  // [warp][parity][group, column]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = lane & (G - 1), grp = lane & ~(G - 1);  // lane in the group, its first lane
  const long w = (long(blockIdx.x) * (blockDim.x >> 5) + warp) * (32 / G) + lane / G;
  const bool mat_ok = w < W, row_ok = mat_ok && i < N;
  const c128* Aw = A + (mat_ok ? w : 0) * strideA + long(i) * N;

  c128 a[NC];
#pragma unroll
  for (int j = 0; j < NC; ++j) a[j] = (row_ok && j < N) ? Aw[j] : cmk(0.0, 0.0);
  int r = i;               // logical row
  c128 piv_i = cmk(1, 0);  // lane k keeps pivot k and its row
  int perm_i = i;
  bool singular = false;

  for (int k = 0; k < N; ++k) {
    const c128 f = a[0];
    // pivot: first max |re|+|im| over the logical rows k..N-1 (NaN counts as 0)
    const bool cand = row_ok && r >= k;
    const double v = cand ? cabs1(f) : 0.0;
    unsigned long long key = (v == v) ? static_cast<unsigned long long>(__double_as_longlong(v)) : 0ull;
    unsigned id = cand ? unsigned(r) * 32u + unsigned(lane) : 0xffffffffu;
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      const unsigned long long ok = __shfl_xor_sync(FULL, key, o);
      const unsigned oid = __shfl_xor_sync(FULL, id, o);
      if (ok > key || (ok == key && oid < id)) {
        key = ok;
        id = oid;
      }
    }
    const bool zero = key == 0ull;
    // a zero (or NaN) column: zero pivot at row k, no interchange; the candidates of a zero key
    // tie, so the first of them is row k itself
    const int pl = mat_ok ? int(id & 31u) : lane, p = mat_ok ? int(id >> 5) : 0;
    const c128 piv = cmk(__shfl_sync(FULL, f.x, pl), __shfl_sync(FULL, f.y, pl));
    const double rden = 1.0 / (piv.x * piv.x + piv.y * piv.y);
    const c128 dinv = cmk(piv.x * rden, -piv.y * rden);
    if (i == k) {
      piv_i = piv;
      perm_i = p;
    }
    singular = singular || zero;
    const bool is_piv = lane == pl;
    c128* row = nullptr;
    if constexpr (SMEM_ROW) {
      row = rows[warp][k & 1] + grp;
      if (is_piv) {
#pragma unroll
        for (int j = 1; j < NC; ++j) row[j] = a[j];
      }
      __syncwarp();
    }
    // logical rows after the interchange
    if (is_piv)
      r = k;
    else if (r == k)
      r = p;
    const c128 gg = cmul(f, dinv), ng = cmk(-gg.x, -gg.y);
    const bool upd = !zero && !is_piv && (INVERT || r > k);
    const bool scl = !zero && is_piv && INVERT;
#pragma unroll
    for (int j = 1; j < NC; ++j) {
      c128 x;
      if constexpr (SMEM_ROW)
        x = row[j];
      else
        x = cmk(__shfl_sync(FULL, a[j].x, pl), __shfl_sync(FULL, a[j].y, pl));
      c128 y = a[j];
      if (upd) {
        y.x = fma(ng.x, x.x, fma(gg.y, x.y, y.x));
        y.y = fma(ng.x, x.y, fma(ng.y, x.x, y.y));
      } else if (scl) {
        y = cmul(x, dinv);
      }
      a[j - 1] = y;
    }
    a[NC - 1] = upd ? ng : (scl ? dinv : cmk(0.0, 0.0));
  }

  // log det: sum_k log(+-U_kk + DBL_MIN) over the group
  c128 l = cmk(0, 0);
  if (row_ok) l = log_pivot(piv_i, perm_i != i);
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    l.x += __shfl_xor_sync(FULL, l.x, o);
    l.y += __shfl_xor_sync(FULL, l.y, o);
  }
  if (mat_ok && i == 0) ovlp[w] = cadd(cmul(post_scale, wrap_imag(cadd(ovlp[w], l))), post_add);
  if (INVERT) {
    // the interchanges, undone on the columns in reverse order: pos = where column i ends
    int pos = i;
    for (int k = N - 1; k >= 0; --k) {
      const int q = __shfl_sync(FULL, perm_i, grp + k);
      if (pos == k)
        pos = q;
      else if (pos == q)
        pos = k;
    }
    c128* Iw = Ainv + (mat_ok ? w : 0) * strideInv + long(r) * N;
#pragma unroll
    for (int j = 0; j < NC; ++j) {  // register j holds column j - (NC - N)
      const int col = j - (NC - N), c = __shfl_sync(FULL, pos, grp + (col > 0 ? col : 0));
      if (row_ok && col >= 0) Iw[c] = singular ? cmk(0.0, 0.0) : a[j];
    }
  }
}

template <int G, int NC>
void launch_gj_warp(cudaStream_t s, const c128* A, long strideA, c128* Ainv, long strideInv,
                    c128* ovlp, int W, int N, bool invert, c128 post_scale, c128 post_add) {
  // single-warp blocks until every SM has a block's worth, so that few matrices spread out
  const int nw = ceil_div(W, 32 / G) < NUM_SMS * GW_WARPS ? 1 : GW_WARPS;
  const int grid = ceil_div(W, nw * (32 / G));
  if (invert)
    gj_warp_kernel<G, NC, true><<<grid, 32 * nw, 0, s>>>(A, strideA, Ainv, strideInv, ovlp, W,
                                                              N, post_scale, post_add);
  else
    gj_warp_kernel<G, NC, false><<<grid, 32 * nw, 0, s>>>(A, strideA, nullptr, 0, ovlp, W, N,
                                                               post_scale, post_add);
}

// ---------------------------------------------------------------------------------------------
// Register-resident Gauss-Jordan / LU for 16 < N <= 32, and for the inverse of few matrices of N > 12
// (a matrix per warp takes longer there: 27 x 27 in a warp's registers leaves too few warps an SM,
// and one matrix of 16 x 16 waits on its own chain).  One CTA of four warps per matrix: lane i holds
// row i and warp h the columns j = h + 4 q of it, in registers (q < QMAX), so a step touches shared
// memory only for the pivot column, the pivot row and the row that moves in the interchange.
// Step k: every warp finds the pivot p (first max |re|+|im| in column k, rows k..N-1, as izamax)
// from the column buffer; the owners of row p write it as it stands with 1 in column k, the owners
// of row k write the old row k; after one barrier every row i != k subtracts g_i times the pivot
// row, g_i = f_i / pivot with f_i its column-k element before the interchange (the multiplier in
// getf2's rounding order), and row p takes the old row k first.  Column k is moved to the column
// buffer and zeroed in the registers at the end of step k-1, so the update leaves -g_i there (the
// in-place Gauss-Jordan inverse); row k becomes the pivot row / pivot.  Without the inverse only
// rows below k are eliminated (plain LU, the same U diagonal).  The row interchanges permute the
// columns of the in-place inverse; they are undone on the way out (columns swapped in reverse step
// order).  Two barriers a step.
// Bound by the chain of a step (pivot search, reciprocal, two barriers); with 89 registers five CTAs
// an SM overlap theirs.  Rows 0..63 on two column classes (half the lanes without a row, 164
// registers, three CTAs) took 139.7 us for the inverses of 1024 matrices of N = 32 and 41.1 for 64
// of them; this form 91.1 and 32.9.
// ---------------------------------------------------------------------------------------------
constexpr int GR_C = 4;  // column classes: warps of a CTA

template <int QMAX, bool INVERT>
__global__ void __launch_bounds__(32 * GR_C, QMAX <= 4 ? 6 : 5)
    gj_reg_kernel(const c128* __restrict__ A, long strideA, c128* __restrict__ Ainv, long strideInv,
                  c128* __restrict__ ovlp, int N, c128 post_scale, c128 post_add) {
  constexpr int C = GR_C;
  __shared__ c128 rowbuf[32];     // pivot row, column k = 1
  __shared__ c128 kbuf[32];       // old row k (moves to row p)
  __shared__ c128 colbuf[2][32];  // column k of every row at step k (buffer k & 1)
  __shared__ c128 piv_val[32];
  __shared__ int perm[32];
  __shared__ int pos[32];
  __shared__ int s_singular;

  const int t = threadIdx.x;
  const int i = t & 31;
  const int h = t >> 5;  // column class: columns j = h + C q
  const bool row_ok = i < N;
  const long w = blockIdx.x;
  const c128* Aw = A + w * strideA;

  c128 a[QMAX];
#pragma unroll
  for (int q = 0; q < QMAX; ++q) {
    const int j = h + C * q;
    a[q] = (row_ok && j < N) ? Aw[long(i) * N + j] : cmk(0.0, 0.0);
  }
  if (h == 0) {
    if (row_ok) colbuf[0][i] = a[0];
    a[0] = cmk(0.0, 0.0);
  }
  if (t == 0) s_singular = 0;
  __syncthreads();

  for (int k = 0; k < N; ++k) {
    const c128* col = colbuf[k & 1];
    // pivot: first max |re|+|im| in column k, rows k..N-1.  Non-negative doubles order as their
    // bit patterns, so the maximum is two warp max-reductions (high, then low word); NaN and rows
    // outside k..N-1 take key 0.  The first row holding the maximum comes from a ballot.
    const bool cand = row_ok && i >= k;
    const double v = cand ? cabs1(col[i]) : 0.0;
    const unsigned long long kl = (v == v) ? static_cast<unsigned long long>(__double_as_longlong(v)) : 0ull;
    const unsigned mhi = __reduce_max_sync(0xffffffffu, unsigned(kl >> 32));
    const unsigned mlo = __reduce_max_sync(0xffffffffu, unsigned(kl >> 32) == mhi ? unsigned(kl) : 0u);
    const unsigned long long kmax = (static_cast<unsigned long long>(mhi) << 32) | mlo;
    const bool zero = (kmax == 0ull);
    // a zero (or NaN) column: every candidate ties, so zero pivot at row k, no interchange
    const int p = __ffs(__ballot_sync(0xffffffffu, cand && kl == kmax)) - 1;
    const c128 piv = col[p];
    // 1/pivot = conj(pivot) / |pivot|^2
    const double rden = 1.0 / (piv.x * piv.x + piv.y * piv.y);
    const c128 dinv = cmk(piv.x * rden, -piv.y * rden);
    if (t == 0) {
      perm[k] = p;
      piv_val[k] = piv;
      if (zero) s_singular = 1;
    }
    if (!zero) {
      // pivot row as it stands (its column k was zeroed in the registers) with 1 in column k
      if (i == p) {
#pragma unroll
        for (int q = 0; q < QMAX; ++q) {
          const int j = h + C * q;
          if (j < N) rowbuf[j] = a[q];
        }
        if (h == (k % C)) rowbuf[k] = cmk(1.0, 0.0);
      }
      if (i == k && p != k) {
#pragma unroll
        for (int q = 0; q < QMAX; ++q) {
          const int j = h + C * q;
          if (j < N) kbuf[j] = a[q];
        }
      }
    }
    __syncthreads();
    c128* nxt = colbuf[(k + 1) & 1];
    const int kn = k + 1;
    if (!zero && row_ok) {
      if (i == k) {
        // row k <- pivot row / pivot (column k: 1/pivot)
        if (INVERT) {
#pragma unroll
          for (int q = 0; q < QMAX; ++q) {
            const int j = h + C * q;
            if (j < N) a[q] = cmul(rowbuf[j], dinv);
          }
        }
      } else if (INVERT || i > k) {
        // row i -= g * pivot row, g = f / pivot (column k: 0 - g = -f/pivot)
        const c128 f = (i == p) ? col[k] : col[i];
        const c128 g = cmul(f, dinv);
        if (i == p) {
#pragma unroll
          for (int q = 0; q < QMAX; ++q) {
            const int j = h + C * q;
            if (j < N) a[q] = kbuf[j];
          }
        }
        const c128 ng = cmk(-g.x, -g.y);
#pragma unroll
        for (int q = 0; q < QMAX; ++q) {
          const int j = h + C * q;
          if (j < N) {
            const c128 r = rowbuf[j];
            a[q].x = fma(ng.x, r.x, fma(g.y, r.y, a[q].x));
            a[q].y = fma(ng.x, r.y, fma(ng.y, r.x, a[q].y));
          }
          // keep the pivot-row loads in groups of eight (bounds the registers they hold)
          if ((q & 7) == 7) asm volatile("" ::: "memory");
        }
      }
    }
    // column k+1 moves to the column buffer for the next pivot search and is zeroed in the
    // registers (warp-uniform branch to its register)
    if (kn < N && h == (kn % C)) {
      switch (kn / C) {
#define GR_CASE(Q)                          \
  case Q:                                   \
    if (Q < QMAX) {                         \
      constexpr int QQ = Q < QMAX ? Q : 0;  \
      if (row_ok) nxt[i] = a[QQ];           \
      a[QQ] = cmk(0.0, 0.0);                \
    }                                       \
    break;
        GR_CASE(0) GR_CASE(1) GR_CASE(2) GR_CASE(3) GR_CASE(4) GR_CASE(5) GR_CASE(6) GR_CASE(7)
#undef GR_CASE
        default:
          break;
      }
    }
    __syncthreads();
  }

  if (t < 32) {
    double sr = 0.0, si = 0.0;
    for (int k = t; k < N; k += 32) {
      const c128 l = log_pivot(piv_val[k], perm[k] != k);
      sr += l.x;
      si += l.y;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      sr += __shfl_xor_sync(0xffffffffu, sr, off);
      si += __shfl_xor_sync(0xffffffffu, si, off);
    }
    if (t == 0) {
      c128 res = cadd(ovlp[w], cmk(sr, si));
      res = wrap_imag(res);
      ovlp[w] = cadd(cmul(post_scale, res), post_add);
    }
  }
  if (INVERT) {
    // at[c] = column of the in-place result that ends in column c (kept in kbuf's memory,
    // free after the last step); pos is its inverse
    int* at = reinterpret_cast<int*>(kbuf);
    if (t < N) at[t] = t;
    __syncthreads();
    if (t == 0)
      for (int k = N - 1; k >= 0; --k) {
        const int q = perm[k];
        const int x = at[k];
        at[k] = at[q];
        at[q] = x;
      }
    __syncthreads();
    if (t < N) pos[at[t]] = t;
    __syncthreads();
    const bool sing = s_singular != 0;
    if (row_ok) {
      c128* Iw = Ainv + w * strideInv + long(i) * N;
#pragma unroll
      for (int q = 0; q < QMAX; ++q) {
        const int j = h + C * q;
        if (j < N) Iw[pos[j]] = sing ? cmk(0.0, 0.0) : a[q];
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Blocked Gauss-Jordan / LU for 32 < N <= 64: one CTA of four warps per matrix, the matrix in shared
// memory, eight columns at a time.
//   panel     warp 0 holds the panel's columns in registers (two rows per lane) and runs eight
//             in-place Gauss-Jordan steps on them alone: partial pivoting (first max |re|+|im|, as
//             izamax) over the rows not yet used, no block barrier;
//   trailing  the steps' product is the identity with the pivot rows' columns replaced by the
//             finished panel E, so every other column becomes A[:, J] + E A[pivot rows, J] (pivot
//             rows: E A[pivot rows, J]), one rank-8 update on the FP64 tensor path by all warps.
// Without the inverse only the columns right of the panel are updated (E of an unused row is
// -A21 A11^{-1}, so the update is the Schur complement).  Rows are interchanged by index only:
// rlog is a row's logical place.  The interchanges permute the columns of the in-place inverse;
// they are undone on the way out.
// What bounds it is the chain of panel steps (pivot search, reciprocal, row broadcast); the CTAs
// of an SM (four at N = 50) overlap theirs with each other's updates.  The form that ran all N
// steps on block barriers, two a step, took 286 us for 1024 matrices of N = 50 (242 us without the
// inverse), this one 176 (114).  Factorising the next panel beside the update (one warp ahead of three)
// took 190 (150): the other CTAs already fill those slots.
// ---------------------------------------------------------------------------------------------
constexpr int GB_THREADS = 128;

__host__ __device__ inline int gb_pitch(int N) { return N | 1; }          // matrix row pitch
__host__ __device__ inline int gb_bpitch(int N) { return (N + 7) / 8 * 8 + 2; }  // pivot-row copy
inline size_t gb_smem(int N) {
  return (size_t(N) * gb_pitch(N) + 8 * size_t(gb_bpitch(N))) * sizeof(c128);
}

template <bool INVERT>
__global__ void __launch_bounds__(GB_THREADS, 4)
    gj_block_kernel(const c128* __restrict__ A, long strideA, c128* Ainv, long strideInv,
                    c128* __restrict__ ovlp, int N, c128 post_scale, c128 post_add) {
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int P = gb_pitch(N), PB = gb_bpitch(N);
  c128* a = reinterpret_cast<c128*>(smem_raw);  // [N][P]
  c128* bc = a + size_t(N) * P;                 // [8][PB] the panel's pivot rows
  __shared__ c128 xrow[2][8];                   // pivot row of the panel, by step parity
  __shared__ c128 piv_val[64];
  __shared__ int perm[64], rlog[64], at[64], pos[64];
  __shared__ int prow[8];                       // physical row of the panel's pivots
  __shared__ unsigned long long s_pivmask;      // ... as a bit mask
  __shared__ int s_singular;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const long w = blockIdx.x;
  const c128* Aw = A + w * strideA;
  for (int e = tid; e < N * N; e += GB_THREADS) {
    const int i = e / N, j = e - i * N;
    a[i * P + j] = Aw[e];
  }
  const int r0 = lane, r1 = lane + 32;  // warp 0: this lane's rows
  const bool ok0 = r0 < N, ok1 = r1 < N;
  int l0 = r0, l1 = r1;                 // their logical places
  bool singular = false;
  __syncthreads();

  for (int k0 = 0; k0 < N; k0 += 8) {
    const int nb = N - k0 < 8 ? N - k0 : 8;
    c128 p0[8], p1[8];
    unsigned long long pivmask = 0ull;
    if (warp == 0) {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        p0[c] = (ok0 && c < nb) ? a[r0 * P + k0 + c] : cmk(0.0, 0.0);
        p1[c] = (ok1 && c < nb) ? a[r1 * P + k0 + c] : cmk(0.0, 0.0);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (j < nb) {
          const int k = k0 + j;
          // first max |re|+|im| of column k over the logical rows k..N-1 (NaN counts as 0)
          const c128 f0 = p0[j], f1 = p1[j];
          const bool c0 = ok0 && l0 >= k, c1 = ok1 && l1 >= k;
          const double v0 = c0 ? cabs1(f0) : 0.0, v1 = c1 ? cabs1(f1) : 0.0;
          const unsigned long long k0_ = (v0 == v0) ? static_cast<unsigned long long>(__double_as_longlong(v0)) : 0ull;
          const unsigned long long k1_ = (v1 == v1) ? static_cast<unsigned long long>(__double_as_longlong(v1)) : 0ull;
          const unsigned long long kl = k1_ > k0_ ? k1_ : k0_;
          const unsigned mhi = __reduce_max_sync(FULL, unsigned(kl >> 32));
          const unsigned mlo = __reduce_max_sync(FULL, unsigned(kl >> 32) == mhi ? unsigned(kl) : 0u);
          const unsigned long long km = (static_cast<unsigned long long>(mhi) << 32) | mlo;
          const unsigned i0 = (c0 && k0_ == km) ? unsigned(l0) * 64u + unsigned(r0) : FULL;
          const unsigned i1 = (c1 && k1_ == km) ? unsigned(l1) * 64u + unsigned(r1) : FULL;
          const unsigned id = __reduce_min_sync(FULL, i0 < i1 ? i0 : i1);
          const int p = int(id >> 6), pr = int(id & 63u);  // logical place and row of the pivot
          const bool zero = km == 0ull;
          const bool m0 = pr == r0, m1 = pr == r1;
          if (m0 || m1) {
#pragma unroll
            for (int c = 0; c < 8; ++c) xrow[j & 1][c] = m0 ? p0[c] : p1[c];
          }
          __syncwarp();
          const c128 piv = xrow[j & 1][j];
          const double rden = 1.0 / (piv.x * piv.x + piv.y * piv.y);
          const c128 dinv = cmk(piv.x * rden, -piv.y * rden);
          // logical rows after the interchange
          if (m0) l0 = k; else if (l0 == k) l0 = p;
          if (m1) l1 = k; else if (l1 == k) l1 = p;
          if (lane == 0) {
            piv_val[k] = piv;
            perm[k] = p;
            prow[j] = pr;
          }
          pivmask |= 1ull << pr;
          singular = singular || zero;
          const c128 g0 = cmul(f0, dinv), g1 = cmul(f1, dinv);
          const bool u0 = !zero && !m0 && (INVERT || l0 > k), u1 = !zero && !m1 && (INVERT || l1 > k);
          const bool s0 = !zero && m0 && INVERT, s1 = !zero && m1 && INVERT;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            if (c == j) continue;
            const c128 x = xrow[j & 1][c];
            if (u0) {
              p0[c].x = fma(-g0.x, x.x, fma(g0.y, x.y, p0[c].x));
              p0[c].y = fma(-g0.x, x.y, fma(-g0.y, x.x, p0[c].y));
            } else if (s0) {
              p0[c] = cmul(x, dinv);
            }
            if (u1) {
              p1[c].x = fma(-g1.x, x.x, fma(g1.y, x.y, p1[c].x));
              p1[c].y = fma(-g1.x, x.y, fma(-g1.y, x.x, p1[c].y));
            } else if (s1) {
              p1[c] = cmul(x, dinv);
            }
          }
          p0[j] = u0 ? cmk(-g0.x, -g0.y) : (s0 ? dinv : cmk(0.0, 0.0));
          p1[j] = u1 ? cmk(-g1.x, -g1.y) : (s1 ? dinv : cmk(0.0, 0.0));
        }
      }
      if (lane == 0) s_pivmask = pivmask;
    }
    __syncthreads();
    // warp 0 stores the finished panel; the others copy the pivot rows' other columns
    const int j_lo = INVERT ? 0 : k0 + 8;
    if (warp == 0) {
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c < nb) {
          // without the inverse a used row takes no further part: its multipliers are zero
          if (ok0) a[r0 * P + k0 + c] = (INVERT || l0 >= k0 + nb) ? p0[c] : cmk(0.0, 0.0);
          if (ok1) a[r1 * P + k0 + c] = (INVERT || l1 >= k0 + nb) ? p1[c] : cmk(0.0, 0.0);
        }
    } else {
      for (int q = warp - 1; q < 8; q += GB_THREADS / 32 - 1)
        for (int j = j_lo + lane; j < PB - 2; j += 32)
          if (j < k0 || j >= k0 + 8)
            bc[q * PB + j] = (q < nb && j < N) ? a[prow[q] * P + j] : cmk(0.0, 0.0);
    }
    __syncthreads();
    const unsigned long long pm = s_pivmask;
    const int nt = (N + 7) / 8, kt = k0 / 8;
    for (int e = warp; e < nt * nt; e += GB_THREADS / 32) {
      const int tc = e / nt, tr = e - tc * nt;
      if (tc == kt || (!INVERT && tc < kt)) continue;
      const int row = tr * 8 + g, col = tc * 8 + 2 * t;
      const bool rok = row < N, keep = rok && !((pm >> row) & 1ull);
      c128* ar = a + (rok ? row : 0) * P;
      double cr[2] = {0.0, 0.0}, ci[2] = {0.0, 0.0};
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (keep && col + h < N) {
          const c128 v = ar[col + h];
          cr[h] = v.x;
          ci[h] = v.y;
        }
#pragma unroll
      for (int kk = 0; kk < 8; kk += 4) {
        const c128 fa = (rok && kk + t < nb) ? ar[k0 + kk + t] : cmk(0.0, 0.0);
        const c128 fb = bc[(kk + t) * PB + tc * 8 + g];
        zmma(cr, ci, fa, fb);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (rok && col + h < N && (INVERT || keep)) ar[col + h] = cmk(cr[h], ci[h]);
    }
    __syncthreads();
  }

  if (warp == 0) {
    if (ok0) rlog[r0] = l0;
    if (ok1) rlog[r1] = l1;
    if (lane == 0) s_singular = singular ? 1 : 0;
    double sr = 0.0, si = 0.0;
    for (int k = lane; k < N; k += 32) {
      const c128 l = log_pivot(piv_val[k], perm[k] != k);
      sr += l.x;
      si += l.y;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      sr += __shfl_xor_sync(FULL, sr, off);
      si += __shfl_xor_sync(FULL, si, off);
    }
    if (lane == 0)
      ovlp[w] = cadd(cmul(post_scale, wrap_imag(cadd(ovlp[w], cmk(sr, si)))), post_add);
  }
  if (INVERT) {
    // at[c] = column of the in-place result that ends in column c; pos is its inverse
    if (tid < N) at[tid] = tid;
    __syncthreads();
    if (tid == 0)
      for (int k = N - 1; k >= 0; --k) {
        const int q = perm[k], x = at[k];
        at[k] = at[q];
        at[q] = x;
      }
    __syncthreads();
    if (tid < N) pos[at[tid]] = tid;
    __syncthreads();
    c128* Iw = Ainv + w * strideInv;
    const bool sing = s_singular != 0;
    for (int e = tid; e < N * N; e += GB_THREADS) {
      const int i = e / N, j = e - i * N;
      Iw[long(rlog[i]) * N + pos[j]] = sing ? cmk(0.0, 0.0) : a[i * P + j];
    }
  }
}

int batched_logdet_inverse(cudaStream_t s, const c128* A, long strideA, c128* Ainv, long strideInv,
                           c128* ovlp, int W, int N, bool invert, c128 post_scale, c128 post_add) {
  if (W <= 0 || N <= 0) return AFQMC_OK;
  if (N <= 64) {
#define GJ_WARP(G, NC)   \
  if (N <= NC) {         \
    launch_gj_warp<G, NC>(s, A, strideA, Ainv, strideInv, ovlp, W, N, invert, post_scale, post_add); \
    return launch_status("gj_warp_kernel"); \
  }
    GJ_WARP(4, 4) GJ_WARP(8, 8) GJ_WARP(16, 12)
    // up to two matrices an SM the inverse takes 16.5 us by a CTA each and 20.6 by a warp (N = 16);
    // 1024 of them 41 (as the CTA form then was) and 21.2.  The LU alone: 18.6 either way.
    if (N <= 16 && invert && W <= 2 * NUM_SMS) {
      gj_reg_kernel<4, true><<<W, 32 * GR_C, 0, s>>>(A, strideA, Ainv, strideInv, ovlp, N,
                                                     post_scale, post_add);
      return launch_status("gj_reg_kernel");
    }
    GJ_WARP(16, 16)
#undef GJ_WARP
    if (N <= 32) {
      if (invert)
        gj_reg_kernel<8, true><<<W, 32 * GR_C, 0, s>>>(A, strideA, Ainv, strideInv, ovlp, N,
                                                       post_scale, post_add);
      else
        gj_reg_kernel<8, false><<<W, 32 * GR_C, 0, s>>>(A, strideA, nullptr, 0, ovlp, N, post_scale,
                                                        post_add);
      return launch_status("gj_reg_kernel");
    }
    const size_t smem = gb_smem(N);
    if (invert) {
      AFQMC_TRY(allow_smem(gj_block_kernel<true>, smem, gb_smem(64)));
      gj_block_kernel<true><<<W, GB_THREADS, smem, s>>>(A, strideA, Ainv, strideInv, ovlp, N,
                                                        post_scale, post_add);
    } else {
      AFQMC_TRY(allow_smem(gj_block_kernel<false>, smem, gb_smem(64)));
      gj_block_kernel<false><<<W, GB_THREADS, smem, s>>>(A, strideA, nullptr, 0, ovlp, N,
                                                         post_scale, post_add);
    }
    return launch_status("gj_block_kernel");
  }
  const int P = invert ? 2 * N : N;
  const int PP = P | 1;
  size_t smem = (size_t(N) * PP + 2 * size_t(P) + 2 * size_t(N)) * sizeof(c128) + N * sizeof(int);
  if (smem > 227 * 1024) {
    set_error_detail("batched_logdet_inverse: N = %d exceeds the shared-memory kernel", N);
    return AFQMC_ERR_UNSUPPORTED;
  }
  if (invert) {
    AFQMC_TRY(allow_smem(gj_logdet_kernel<true>, smem, GJ_SMEM_MAX));
    gj_logdet_kernel<true><<<W, GJ_THREADS, smem, s>>>(A, strideA, Ainv, strideInv, ovlp, N,
                                                       post_scale, post_add);
  } else {
    AFQMC_TRY(allow_smem(gj_logdet_kernel<false>, smem, GJ_SMEM_MAX));
    gj_logdet_kernel<false><<<W, GJ_THREADS, smem, s>>>(A, strideA, nullptr, 0, ovlp, N,
                                                        post_scale, post_add);
  }
  return launch_status("gj_logdet_kernel");
}

// ---------------------------------------------------------------------------------------------
// Mixed density matrix / log overlap
// ---------------------------------------------------------------------------------------------
int overlap_matrices(cudaStream_t s, const c128* PsiT, const c128* S, long ldS, c128* T, int W,
                     int M, int N, const double* PsiT_r) {
  // T_w = PsiT (N x M) * S_w (M x N)   (math::product(A,B,TNN), density_matrix.hpp:142)
  GemmParams p{};
  p.m = N; p.n = N; p.k = M;
  p.A = PsiT_r ? (const void*)PsiT_r : (const void*)PsiT; p.lda = M; p.strideA = 0;
  p.B = S; p.ldb = N; p.strideB = ldS;
  p.C = T; p.ldc = N; p.strideC = long(N) * N;
  p.alpha = cmk(1, 0); p.beta = cmk(0, 0);
  return zgemm(s, W, GN, PsiT_r != nullptr, GN, false, p);
}

int log_overlap(cudaStream_t s, const c128* PsiT, const c128* S, long ldS, c128* ovlp, int W,
                int M, int N, c128* work_T, c128 post_scale, c128 post_add,
                const double* PsiT_r) {
  if (N == 0) return AFQMC_OK;
  AFQMC_TRY(overlap_matrices(s, PsiT, S, ldS, work_T, W, M, N, PsiT_r));
  return batched_logdet_inverse(s, work_T, long(N) * N, nullptr, 0, ovlp, W, N, false, post_scale,
                                post_add);
}

int mixed_density_matrix(cudaStream_t s, const c128* PsiT, const c128* S, long ldS, c128* G,
                         long ldG, c128* ovlp, int W, int M, int N, bool compact, c128* work_T,
                         c128* work_NM, c128 post_scale, c128 post_add,
                         const double* PsiT_r) {
  if (N == 0) return AFQMC_OK;
  AFQMC_TRY(overlap_matrices(s, PsiT, S, ldS, work_T, W, M, N, PsiT_r));
  AFQMC_TRY(batched_logdet_inverse(s, work_T, long(N) * N, work_T, long(N) * N, ovlp, W, N, true,
                                   post_scale, post_add));
  // C = TNN^T * S^T  (product<'T','T'>, density_matrix.hpp:576): [N x M]
  c128* Cc = compact ? G : work_NM;
  long ldc_w = compact ? ldG : long(N) * M;
  GemmParams p{};
  p.m = N; p.n = M; p.k = N;
  p.A = work_T; p.lda = N; p.strideA = long(N) * N;
  p.B = S; p.ldb = N; p.strideB = ldS;
  p.C = Cc; p.ldc = M; p.strideC = ldc_w;
  p.alpha = cmk(1, 0); p.beta = cmk(0, 0);
  AFQMC_TRY(zgemm(s, W, GT, false, GT, false, p));
  if (compact) return AFQMC_OK;
  // full G = PsiT^T * C  (product<'T'>(A,TNM,C), density_matrix.hpp:584): [M x M]
  GemmParams q{};
  q.m = M; q.n = M; q.k = N;
  q.A = PsiT; q.lda = M; q.strideA = 0;
  q.B = work_NM; q.ldb = M; q.strideB = long(N) * M;
  q.C = G; q.ldc = M; q.strideC = ldG;
  q.alpha = cmk(1, 0); q.beta = cmk(0, 0);
  return zgemm(s, W, GT, false, GN, false, q);
}

// ---------------------------------------------------------------------------------------------
// Taylor propagation: S <- P1 exp_T(i V) P1 S  (propagate.hpp:41-70, 238-298)
// work1/work2/work3: [W][M][N] each.
// ---------------------------------------------------------------------------------------------
int propagate(cudaStream_t s, const void* P1, bool p1_real, const c128* V, long strideV, c128* S,
              long ldS, int W, int M, int N, int order, c128* work1, c128* work2, c128* work3) {
  if (N == 0 || W == 0) return AFQMC_OK;
  if (taylor_c128_fits(W, M, N))
    return taylor_c128(s, P1, p1_real, V, strideV, S, ldS, W, M, N, order);
  const long sMN = long(M) * N;
  // T0 = P1 * S into work2, and the running sum TMN = T0 into work1
  GemmParams p{};
  p.m = M; p.n = N; p.k = M;
  p.A = P1; p.lda = M; p.strideA = 0;
  p.B = S; p.ldb = N; p.strideB = ldS;
  p.C = work2; p.ldc = N; p.strideC = sMN;
  p.alpha = cmk(1, 0); p.beta = cmk(0, 0);
  p.D = work1; p.ldd = N; p.strideD = sMN; p.d_store = true;
  AFQMC_TRY(zgemm(s, W, GN, p1_real, GN, false, p));
  // T_n = (i/n) V T_{n-1};  TMN += T_n   (apply_expM<'N'>)
  c128* Tprev = work2;
  c128* Tnext = work3;
  for (int n = 1; n <= order; ++n) {
    GemmParams q{};
    q.m = M; q.n = N; q.k = M;
    q.A = V; q.lda = M; q.strideA = strideV;
    q.B = Tprev; q.ldb = N; q.strideB = sMN;
    q.C = Tnext; q.ldc = N; q.strideC = sMN;
    q.alpha = cmk(0.0, 1.0 / double(n)); q.beta = cmk(0, 0);
    q.D = work1; q.ldd = N; q.strideD = sMN; q.d_store = false;
    AFQMC_TRY(zgemm(s, W, GN, false, GN, false, q));
    c128* t = Tprev;
    Tprev = Tnext;
    Tnext = t;
  }
  // S = P1 * TMN
  GemmParams r{};
  r.m = M; r.n = N; r.k = M;
  r.A = P1; r.lda = M; r.strideA = 0;
  r.B = work1; r.ldb = N; r.strideB = sMN;
  r.C = S; r.ldc = N; r.strideC = ldS;
  r.alpha = cmk(1, 0); r.beta = cmk(0, 0);
  return zgemm(s, W, GN, p1_real, GN, false, r);
}

}  // namespace afqmc
