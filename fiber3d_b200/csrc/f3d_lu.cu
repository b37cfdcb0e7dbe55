// Batched LU factorisation with partial pivoting, and the matching solve,
// for many small dense FP64 systems of uneven size in ONE persistent launch
// each: the per-fiber (4N x 4N) and per-body ((3Nb+6)^2) blocks of the
// block-diagonal preconditioner.
//
// Replaces, per block, scipy.linalg.lu_factor / lu_solve as called by
// build_block_diagonal_lu_preconditioner_fiber (tstep/tstep_utils.py:1405-1419),
// build_block_diagonal_preconditioner_body (tstep_utils.py:1341-1386) and
// P_inv (tstep/tstep.py:950-994).  Pivot convention as LAPACK getrf: at step
// i, row i was swapped with row piv[i] (0-based here), the pivot being the
// first entry of largest magnitude in the column.
//
// Factor: one CTA per matrix, CTAs take matrices from a queue (atomic counter,
// host-supplied order, largest first) until it is empty.  Blocked
// right-looking algorithm, two kernels:
//  * blocks of up to 256 rows (lu_tc_kernel): 16-column panels, the rows of
//    a panel in registers, one barrier per pivot, the trailing update on the
//    FP64 tensor cores; described at the kernel;
//  * larger blocks, and explicit panel widths (batched_lu_factor_kernel): an
//    NB-column panel held in shared memory:
//   1. panel (n-k0) x NB loaded to shared memory (column-major), unblocked
//      LU with pivot search by block argmax reduction;
//   2. panel written back, its row swaps applied to the other columns;
//   3. U12 = L11^-1 A12 (one thread per column, NB unrolled);
//   4. A22 -= L21 U12 in column chunks of 64 staged in shared memory,
//      4x2 register tiles.
// The trailing matrix stays in global memory; it is L2-resident while the CTA
// works on it.
// Solve: one CTA per system (persistent over systems), right-hand side in
// shared memory, substitution by blocks of 32 unknowns; batches of many small
// systems by one warp per system.
#include <algorithm>
#include <climits>

#include "f3d_common.cuh"

namespace f3d {

constexpr int kLuThreads = 256;
constexpr int kChunk = 64;  // columns of U12 staged per GEMM chunk

struct LuArgs {
  double *A;
  const int64_t *moff;   // matrix offsets (elements)
  const int64_t *voff;   // vector/pivot offsets (elements)
  const int32_t *sizes;
  const int32_t *order;  // processing order or nullptr
  int32_t *piv;
  int32_t *info;
  unsigned *queue;       // [2] work counter, finished-CTA counter (zero on entry and exit)
  int count;
};

template <int NB>
__device__ void lu_factor_one(double *__restrict__ A, int n, int32_t *__restrict__ piv,
                              int32_t *info, double *smem) {
  double *P = smem;                                // panel, column-major, m rows
  double *U = smem + static_cast<size_t>(n) * NB;  // U12 chunk: NB x kChunk (row-major)
  __shared__ int s_piv[NB];
  __shared__ double s_val[kLuThreads / 32];
  __shared__ int s_idx[kLuThreads / 32];
  __shared__ int s_info;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  if (tid == 0) s_info = 0;

  for (int k0 = 0; k0 < n; k0 += NB) {
    const int nb = min(NB, n - k0);
    const int m = n - k0;
    for (int idx = tid; idx < m * nb; idx += kLuThreads) {
      const int r = idx / nb, c = idx - r * nb;
      P[c * m + r] = A[static_cast<int64_t>(k0 + r) * n + k0 + c];
    }
    __syncthreads();
    for (int j = 0; j < nb; ++j) {
      // argmax |P[j:m, j]|, first index on ties
      double best = -1.0;
      int bi = m;
      for (int r = j + tid; r < m; r += kLuThreads) {
        const double v = fabs(P[j * m + r]);
        if (v > best) { best = v; bi = r; }
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, best, off);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
        if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
      }
      if (lane == 0) { s_val[warp] = best; s_idx[warp] = bi; }
      __syncthreads();
      if (tid == 0) {
        double bv = s_val[0];
        int bix = s_idx[0];
        for (int w = 1; w < kLuThreads / 32; ++w) {
          if (s_val[w] > bv || (s_val[w] == bv && s_idx[w] < bix)) { bv = s_val[w]; bix = s_idx[w]; }
        }
        if (bix >= m) bix = j;
        s_piv[j] = bix;
        if (P[j * m + bix] == 0.0 && s_info == 0) s_info = k0 + j + 1;
      }
      __syncthreads();
      const int p = s_piv[j];
      if (p != j) {
        for (int c = tid; c < nb; c += kLuThreads) {
          const double t = P[c * m + j];
          P[c * m + j] = P[c * m + p];
          P[c * m + p] = t;
        }
      }
      __syncthreads();
      const double pv = P[j * m + j];
      if (pv != 0.0) {
        for (int r = j + 1 + tid; r < m; r += kLuThreads) P[j * m + r] /= pv;
      }
      __syncthreads();
      const int mr = m - j - 1, nc = nb - j - 1;
      for (int idx = tid; idx < mr * nc; idx += kLuThreads) {
        const int c = j + 1 + idx / mr, r = j + 1 + idx % mr;
        P[c * m + r] -= P[j * m + r] * P[c * m + j];
      }
      __syncthreads();
    }
    for (int idx = tid; idx < m * nb; idx += kLuThreads) {
      const int r = idx / nb, c = idx - r * nb;
      A[static_cast<int64_t>(k0 + r) * n + k0 + c] = P[c * m + r];
    }
    if (tid < nb) piv[k0 + tid] = k0 + s_piv[tid];
    // Row swaps on the columns outside the panel.  Thread t owns the same
    // columns for every j, so the swaps stay in order without barriers.
    const int nout = n - nb;
    for (int j = 0; j < nb; ++j) {
      const int p = s_piv[j];
      if (p == j) continue;
      for (int c = tid; c < nout; c += kLuThreads) {
        const int col = c < k0 ? c : c + nb;
        double *a = A + static_cast<int64_t>(k0 + j) * n + col;
        double *b = A + static_cast<int64_t>(k0 + p) * n + col;
        const double t = *a;
        *a = *b;
        *b = t;
      }
    }
    __syncthreads();
    const int n2 = n - k0 - nb;
    if (n2 > 0) {
      // U12 = L11^-1 A12 (unit lower L11 = P[0:nb, 0:nb])
      for (int col = k0 + nb + tid; col < n; col += kLuThreads) {
        double u[NB];
#pragma unroll
        for (int r = 0; r < NB; ++r) u[r] = (r < nb) ? A[static_cast<int64_t>(k0 + r) * n + col] : 0.0;
#pragma unroll
        for (int r = 1; r < NB; ++r) {
#pragma unroll
          for (int q = 0; q < NB; ++q)
            if (q < r && r < nb) u[r] -= P[q * m + r] * u[q];
        }
#pragma unroll
        for (int r = 0; r < NB; ++r)
          if (r < nb) A[static_cast<int64_t>(k0 + r) * n + col] = u[r];
      }
      __syncthreads();
      // A22 -= L21 U12, chunked over columns
      const int m2 = m - nb;
      for (int c0 = 0; c0 < n2; c0 += kChunk) {
        const int cw = min(kChunk, n2 - c0);
        for (int idx = tid; idx < nb * kChunk; idx += kLuThreads) {
          const int l = idx / kChunk, c = idx - l * kChunk;
          U[l * kChunk + c] = (c < cw) ? A[static_cast<int64_t>(k0 + l) * n + k0 + nb + c0 + c] : 0.0;
        }
        __syncthreads();
        // thread tile: 4 rows x 2 columns; 32 column pairs x 8 row groups
        const int cp = tid & 31;        // column pair
        const int rg = tid >> 5;        // row group (warp)
        const int cA = 2 * cp, cB = 2 * cp + 1;
        for (int r0 = 4 * rg; r0 < m2; r0 += 4 * (kLuThreads / 32)) {
          double acc[4][2];
#pragma unroll
          for (int a = 0; a < 4; ++a) { acc[a][0] = 0.0; acc[a][1] = 0.0; }
#pragma unroll 4
          for (int l = 0; l < nb; ++l) {
            const double uA = U[l * kChunk + cA], uB = U[l * kChunk + cB];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
              const int r = r0 + a;
              const double lv = (r < m2) ? P[l * m + nb + r] : 0.0;
              acc[a][0] = fma(lv, uA, acc[a][0]);
              acc[a][1] = fma(lv, uB, acc[a][1]);
            }
          }
#pragma unroll
          for (int a = 0; a < 4; ++a) {
            const int r = r0 + a;
            if (r < m2) {
              double *row = A + static_cast<int64_t>(k0 + nb + r) * n + k0 + nb + c0;
              if (cA < cw) row[cA] -= acc[a][0];
              if (cB < cw) row[cB] -= acc[a][1];
            }
          }
        }
        __syncthreads();
      }
    }
  }
  __syncthreads();
  if (tid == 0) *info = s_info;
}

template <int NB>
__global__ void __launch_bounds__(kLuThreads) batched_lu_factor_kernel(const LuArgs a) {
  extern __shared__ __align__(16) double lu_smem[];
  __shared__ int s_item;
  while (true) {
    if (threadIdx.x == 0) s_item = static_cast<int>(atomicAdd(&a.queue[0], 1u));
    __syncthreads();
    const int item = s_item;
    __syncthreads();
    if (item >= a.count) break;
    const int b = a.order ? a.order[item] : item;
    const int n = a.sizes[b];
    if (n > 0) lu_factor_one<NB>(a.A + a.moff[b], n, a.piv + a.voff[b], a.info + b, lu_smem);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&a.queue[1], 1u) == gridDim.x - 1) {
      a.queue[0] = 0u;
      a.queue[1] = 0u;
    }
  }
}

// ---------------------------------------------------- blocks of up to 256 --
// What bounds the factorisation of blocks this small is the chain of n
// dependent pivot steps, not the 2/3 n^3 flops, so the kernel shortens a
// step and keeps several blocks in flight per SM:
//  * A panel is 16 columns.  Thread t holds the panel entries of the row at
//    position k0 + t in registers, so a step is one warp
//    reduction (the leading words of the magnitudes; the rest of the key
//    only among rows that tie), a post of each warp's best row, one barrier
//    and at most 15 independent FMAs per row.
//  * Rows are not exchanged: each carries its position, which a pivot swap
//    changes, and `phys` maps positions to rows.  The pivot is the first
//    position of largest magnitude, LAPACK's choice.  The rows move to their
//    positions once, in a pass at the end.
//  * Positions are also the compact index of the rows still to be reduced:
//    the trailing update gathers them by `phys`, 16 x 32 outputs per warp
//    with one m16n8k16 step per 16 x 8 tile, operands from the panel and U12
//    in shared memory, the matrix itself from L2.
// 256 threads, 80 registers and, up to 224 rows, at most 70 KB per CTA leave three
// blocks per SM, whose pivot chains overlap; above (78 KB with 256 rows) two.  (128 threads with two rows each: 1.95 ms
// on the blocks below; every thread scanning the warps' keys and forming the
// pivot's reciprocal after the barrier: 1.54 ms; 64-bit keys posted in three
// words: 1.37 ms.)  Measured on 2000 blocks of 64-256 rows (7.2 Gflop):
// 1.34 ms, against 5.95 ms for the kernel below with its default panel of 32,
// 2.38 ms with 16 and 3.18 ms with 8; on 2000 blocks of 128 rows 0.64 ms
// against 1.53 ms (16).  One block of 256 rows alone takes 0.30 ms, 0.99 ms
// before.
constexpr int kLtThreads = 256;
constexpr int kLtWarps = kLtThreads / 32;
constexpr int kLtNB = 16;
constexpr int kLtMax = kLtThreads;
constexpr int kLtLS = kLtNB + 4;  // panel row stride (doubles): A-fragment reads 4g + t apart

static __host__ __device__ constexpr int lt_us(int n) { return (n + 31) / 32 * 32 + 4; }  // U12 row stride

static size_t lt_smem(int max_n) {
  return (static_cast<size_t>((max_n + 15) / 16 * 16) * kLtLS + static_cast<size_t>(kLtNB) * lt_us(max_n)) *
         sizeof(double);
}

struct LtShared {
  __align__(16) double cand[2][kLtWarps][kLtNB];  // each warp's best row, by step parity
  uint4 post[2][kLtWarps];                        // its candidate's trailing word, position, and reciprocal
  unsigned hi[2][kLtWarps];                       // the candidate's key
  __align__(16) double l11[kLtNB][kLtNB];         // column-major unit lower triangle of the panel
  int piv[kLtNB];
  int phys[kLtMax];
  int info, item;
};

template <bool VEC>
__device__ __forceinline__ void lt_factor_one(double *__restrict__ A, int n, int32_t *__restrict__ piv,
                                              int32_t *__restrict__ info, double *Ls, double *Us, int us,
                                              LtShared &S) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < n) S.phys[tid] = tid;
  if (tid == 0) S.info = 0;
  __syncthreads();
  for (int k0 = 0; k0 < n; k0 += kLtNB) {
    const int nb = min(kLtNB, n - k0), m = n - k0;
    const int nact = (m + 31) / 32;  // warps with rows
    if (warp < nact) {
      double v[kLtNB];
      const bool live = tid < m;
      bool done = !live;
      int pos = live ? k0 + tid : INT_MAX;
      const int row = live ? S.phys[pos] : 0;
      double *const a = A + static_cast<int64_t>(row) * n + k0;
#pragma unroll
      for (int j = 0; j < kLtNB; ++j) v[j] = 0.0;
      if (live) {
        if (VEC) {
#pragma unroll
          for (int j = 0; j < kLtNB; j += 2)
            if (j < nb) {
              const double2 w = *reinterpret_cast<const double2 *>(a + j);
              v[j] = w.x;
              v[j + 1] = w.y;
            }
        } else {
#pragma unroll
          for (int j = 0; j < kLtNB; ++j)
            if (j < nb) v[j] = a[j];
        }
      }
#pragma unroll
      for (int jj = 0; jj < kLtNB; ++jj) {
        if (jj >= nb) break;
        const int par = jj & 1;
        // this thread's candidate: 0 none, 1 a NaN (chosen only if every
        // candidate is one), else the leading word of |a| plus 2
        const unsigned mag = static_cast<unsigned>(__double2hiint(v[jj])) & 0x7fffffffu;
        const bool nan = v[jj] != v[jj];
        const unsigned hi = done ? 0u : (nan ? 1u : mag + 2u), lo = nan ? 0u : __double2loint(v[jj]);
        // the candidate's reciprocal, beside the search (no branch whatever the
        // row holds): l = v / d is formed from it with one residual correction
        // (Markstein); pivots near the ends of the range divide instead
        const double rcp = reciprocal(v[jj]);
        const unsigned hmax = __reduce_max_sync(0xffffffffu, hi);
        bool best = hi == hmax;
        const unsigned all = __ballot_sync(0xffffffffu, best);
        if (all & (all - 1u)) {  // equal leading words: the trailing ones, then the position
          const unsigned lmax = __reduce_max_sync(0xffffffffu, best ? lo : 0u);
          best = best && lo == lmax;
          const int pmin = __reduce_min_sync(0xffffffffu, best ? pos : INT_MAX);
          best = best && pos == pmin;
        }
        if (best) {  // one lane (a warp with no candidate left posts key 0, which never wins)
          S.hi[par][warp] = hi;
          S.post[par][warp] = make_uint4(lo, static_cast<unsigned>(pos), static_cast<unsigned>(__double2loint(rcp)),
                                         static_cast<unsigned>(__double2hiint(rcp)));
#pragma unroll
          for (int j = jj & ~1; j < kLtNB; j += 2)
            *reinterpret_cast<double2 *>(&S.cand[par][warp][j]) = make_double2(v[j], v[j + 1]);
        }
        asm volatile("bar.sync 1, %0;" ::"r"(32 * nact) : "memory");
        // the best warp: lane w looks at warp w's post
        const unsigned wh = (lane & 7) < nact ? S.hi[par][lane & 7] : 0u;
        const unsigned whmax = __reduce_max_sync(0xffffffffu, wh);
        unsigned ties = __ballot_sync(0xffffffffu, wh == whmax) & ((1u << nact) - 1u);
        int bw = __ffs(ties) - 1;
        while (ties &= ties - 1u) {  // equal leading words: the rest of the key, then the position
          const int w = __ffs(ties) - 1;
          const uint4 pw = S.post[par][w], pb = S.post[par][bw];
          if (pw.x > pb.x || (pw.x == pb.x && static_cast<int>(pw.y) < static_cast<int>(pb.y))) bw = w;
        }
        const uint4 post = S.post[par][bw];
        const int pp = static_cast<int>(post.y);
        const double *prow = S.cand[par][bw];
        const double d = prow[jj], rd = __hiloint2double(static_cast<int>(post.w), static_cast<int>(post.z));
        const bool plain = fabs(d) >= 1e-290 && fabs(d) <= 1e290;
        const int k = k0 + jj;
        if (tid == 0) {
          S.piv[jj] = pp;
          if (d == 0.0 && S.info == 0) S.info = k + 1;
        }
        if (pos == pp) {  // the pivot row
          pos = k;
          done = true;
        } else if (pos == k) {
          pos = pp;
        }
        if (!done) {
          double l = v[jj];
          if (plain) {
            const double l0 = l * rd;
            l = fma(fma(-l0, d, l), rd, l0);
          } else if (d != 0.0) {
            l /= d;
          }
          v[jj] = l;
#pragma unroll
          for (int j = jj + 1; j < kLtNB; ++j) v[j] = fma(-l, prow[j], v[j]);
        }
      }
      if (live) {
        if (VEC) {
#pragma unroll
          for (int j = 0; j < kLtNB; j += 2)
            if (j < nb) *reinterpret_cast<double2 *>(a + j) = make_double2(v[j], v[j + 1]);
        } else {
#pragma unroll
          for (int j = 0; j < kLtNB; ++j)
            if (j < nb) a[j] = v[j];
        }
        S.phys[pos] = row;
        const int p = pos - k0;
        if (p >= kLtNB) {
#pragma unroll
          for (int j = 0; j < kLtNB; j += 2)
            *reinterpret_cast<double2 *>(&Ls[(p - kLtNB) * kLtLS + j]) = make_double2(v[j], v[j + 1]);
        } else {
#pragma unroll
          for (int j = 0; j < kLtNB; ++j) S.l11[j][p] = v[j];
        }
      }
    }
    __syncthreads();
    if (tid < nb) piv[k0 + tid] = S.piv[tid];
    const int n2 = m - nb;
    if (n2 <= 0) break;
    double *A2 = A + k0 + kLtNB;  // the trailing columns of row 0
    // U12 = L11^-1 A12, one column per thread
    const int ncol = (n2 + 31) / 32 * 32;
    for (int c = tid; c < ncol; c += kLtThreads) {
      asm volatile("" ::: "memory");  // L11 is read again for each column, not kept in registers
      double u[kLtNB];
#pragma unroll
      for (int i = 0; i < kLtNB; ++i) u[i] = c < n2 ? A2[static_cast<int64_t>(S.phys[k0 + i]) * n + c] : 0.0;
#pragma unroll
      for (int i = 0; i < kLtNB - 1; ++i) {
#pragma unroll
        for (int r = i + 1; r < kLtNB; ++r) u[r] = fma(-S.l11[i][r], u[i], u[r]);
      }
#pragma unroll
      for (int i = 0; i < kLtNB; ++i) {
        Us[i * us + c] = u[i];
        if (i > 0 && c < n2) A2[static_cast<int64_t>(S.phys[k0 + i]) * n + c] = u[i];
      }
    }
    __syncthreads();
    // A22 -= L21 U12
    const int g = lane >> 2, t = lane & 3;
    const int rts = (n2 + 15) / 16, items = rts * (ncol / 32);
    for (int w = warp; w < items; w += kLtWarps) {
      const int rt = w % rts, c0 = 32 * (w / rts);
      const int r0 = 16 * rt + g, r1 = r0 + 8;
      double *x0 = A2 + static_cast<int64_t>(S.phys[k0 + kLtNB + min(r0, n2 - 1)]) * n + c0 + 2 * t;
      double *x1 = A2 + static_cast<int64_t>(S.phys[k0 + kLtNB + min(r1, n2 - 1)]) * n + c0 + 2 * t;
      double x[4][4];
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        const int c = c0 + 8 * ni + 2 * t;
        if (VEC) {
          double2 y0 = make_double2(0.0, 0.0), y1 = y0;
          if (c < n2) {
            y0 = *reinterpret_cast<const double2 *>(x0 + 8 * ni);
            y1 = *reinterpret_cast<const double2 *>(x1 + 8 * ni);
          }
          x[ni][0] = y0.x, x[ni][1] = y0.y, x[ni][2] = y1.x, x[ni][3] = y1.y;
        } else {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            x[ni][e] = c + e < n2 ? x0[8 * ni + e] : 0.0;
            x[ni][2 + e] = c + e < n2 ? x1[8 * ni + e] : 0.0;
          }
        }
      }
      double af[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) af[q] = -Ls[(r0 + 8 * (q & 1)) * kLtLS + t + 4 * (q >> 1)];
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        double bf[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) bf[j] = Us[(t + 4 * j) * us + c0 + 8 * ni + g];
        mma_f64_16816(x[ni], af, bf);
        const int c = c0 + 8 * ni + 2 * t;
        if (VEC) {
          if (c < n2) {
            if (r0 < n2) *reinterpret_cast<double2 *>(x0 + 8 * ni) = make_double2(x[ni][0], x[ni][1]);
            if (r1 < n2) *reinterpret_cast<double2 *>(x1 + 8 * ni) = make_double2(x[ni][2], x[ni][3]);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            if (c + e < n2 && r0 < n2) x0[8 * ni + e] = x[ni][e];
            if (c + e < n2 && r1 < n2) x1[8 * ni + e] = x[ni][2 + e];
          }
        }
      }
    }
    __syncthreads();
  }
  // rows to their positions, 16 columns at a time through shared memory
  // (eight threads per row)
  const int cc = 2 * (tid & 7);
  for (int c0 = 0; c0 < n; c0 += 16) {
    const int c = c0 + cc;
    if (c < n) {
#pragma unroll 8
      for (int p = tid >> 3; p < n; p += kLtThreads / 8) {
        const double *a = A + static_cast<int64_t>(S.phys[p]) * n + c;
        if (VEC) {
          *reinterpret_cast<double2 *>(&Ls[p * kLtLS + cc]) = *reinterpret_cast<const double2 *>(a);
        } else {
          Ls[p * kLtLS + cc] = a[0];
          if (c + 1 < n) Ls[p * kLtLS + cc + 1] = a[1];
        }
      }
    }
    __syncthreads();
    if (c < n) {
#pragma unroll 4
      for (int p = tid >> 3; p < n; p += kLtThreads / 8) {
        if (S.phys[p] == p) continue;
        double *a = A + static_cast<int64_t>(p) * n + c;
        if (VEC) {
          *reinterpret_cast<double2 *>(a) = *reinterpret_cast<const double2 *>(&Ls[p * kLtLS + cc]);
        } else {
          a[0] = Ls[p * kLtLS + cc];
          if (c + 1 < n) a[1] = Ls[p * kLtLS + cc + 1];
        }
      }
    }
    // the threads that read an entry of Ls here are the ones that write it next
  }
  if (tid == 0) *info = S.info;
  __syncthreads();
}

__global__ void __launch_bounds__(kLtThreads, 3) lu_tc_kernel(const LuArgs a, int max_n) {
  extern __shared__ __align__(16) double lu_smem[];
  __shared__ LtShared S;
  double *Ls = lu_smem;
  double *Us = Ls + (max_n + 15) / 16 * 16 * kLtLS;
  const int us = lt_us(max_n);
  while (true) {
    if (threadIdx.x == 0) S.item = static_cast<int>(atomicAdd(&a.queue[0], 1u));
    __syncthreads();
    const int item = S.item;
    if (item >= a.count) break;
    const int b = a.order ? a.order[item] : item;
    const int n = a.sizes[b];
    double *A = a.A + a.moff[b];
    if (n > 0) {
      // 16-byte accesses where every row starts on a 16-byte boundary
      if ((n & 1) == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0)
        lt_factor_one<true>(A, n, a.piv + a.voff[b], a.info + b, Ls, Us, us, S);
      else
        lt_factor_one<false>(A, n, a.piv + a.voff[b], a.info + b, Ls, Us, us, S);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&a.queue[1], 1u) == gridDim.x - 1) {
      a.queue[0] = 0u;
      a.queue[1] = 0u;
    }
  }
}

struct LuSolveArgs {
  const double *LU;
  const int64_t *moff, *voff;
  const int32_t *sizes;
  const int32_t *order;
  const int32_t *piv;
  double *x;  // right-hand sides in, solutions out (packed by voff)
  unsigned *queue;
  int count;
  int max_n;
};

// Substitution by blocks of 32 unknowns: one warp solves the block's 32 x 32
// triangle (from shared memory, a lane per row, the unknowns handed on by
// shuffles), then the CTA takes the block's 32 columns out of the rows that
// remain, eight lanes per row.  A block of the triangle is fetched while the
// rows of the one before are updated.  Reading the factors once (8 n^2
// bytes) bounds it; several CTAs per SM hide the two short chains.  2000
// blocks of 64-256 rows: 192 us (0.43 GB), against 754 us for a warp per
// system with a dot product and five shuffles per unknown.
constexpr int kSvThreads = 128;
constexpr int kSvB = 32;
constexpr int kSvTS = kSvB + 1;  // row stride of the staged triangle

__global__ void __launch_bounds__(kSvThreads) batched_lu_solve_kernel(const LuSolveArgs a) {
  extern __shared__ __align__(16) double sv_smem[];
  double *y = sv_smem;                       // [max_n]
  double *T = y + (a.max_n + 1) / 2 * 2;     // [32][33]
  int *pv = reinterpret_cast<int *>(T + kSvB * kSvTS + 1);  // [max_n]
  __shared__ int s_item;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  while (true) {
    if (tid == 0) s_item = static_cast<int>(atomicAdd(&a.queue[0], 1u));
    __syncthreads();
    const int item = s_item;
    if (item >= a.count) break;
    const int b = a.order ? a.order[item] : item;
    const int n = a.sizes[b];
    const double *L = a.LU + a.moff[b];
    double *x = a.x + a.voff[b];
    const int nblk = (n + kSvB - 1) / kSvB;
    // the 32 x 32 diagonal block at k0, eight entries per thread (0 outside)
    auto fetch = [&](int k0, double (&d)[8]) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = warp + 4 * i;
        d[i] = (k0 + r < n && k0 + lane < n) ? L[static_cast<int64_t>(k0 + r) * n + k0 + lane] : 0.0;
      }
    };
    auto stage = [&](const double (&d)[8]) {
#pragma unroll
      for (int i = 0; i < 8; ++i) T[(warp + 4 * i) * kSvTS + lane] = d[i];
    };
    // y[r] -= sum_j L[r][k0 + j] y[k0 + j], j < kw, for rows [r0, r1)
    const bool vec = (n & 1) == 0 && (reinterpret_cast<uintptr_t>(L) & 15) == 0;
    auto update = [&](int k0, int kw, int r0, int r1) {
      const int sub = tid & 7;
      double yv[2][2];  // the unknowns of this lane's columns 16 h + 2 sub, + 1 (0 past the block)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int j = 16 * h + 2 * sub + e;
          yv[h][e] = j < kw ? y[k0 + j] : 0.0;
        }
      for (int rb = r0; rb < r1; rb += 4 * (kSvThreads / 8)) {  // four rows per lane group at a time
        double2 w[4][2];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = rb + (tid >> 3) + i * (kSvThreads / 8);
          const double *row = L + static_cast<int64_t>(r) * n + k0;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int j = 16 * h + 2 * sub;
            w[i][h] = make_double2(0.0, 0.0);
            if (r < r1) {
              if (vec && j + 1 < kw) {
                w[i][h] = *reinterpret_cast<const double2 *>(row + j);
              } else {
                if (j < kw) w[i][h].x = row[j];
                if (j + 1 < kw) w[i][h].y = row[j + 1];
              }
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          double s = fma(w[i][0].x, yv[0][0],
                         fma(w[i][0].y, yv[0][1], fma(w[i][1].x, yv[1][0], w[i][1].y * yv[1][1])));
#pragma unroll
          for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
          const int r = rb + (tid >> 3) + i * (kSvThreads / 8);
          if (sub == 0 && r < r1) y[r] -= s;
        }
      }
    };
    double d[8];
    fetch(0, d);
    for (int i = tid; i < n; i += kSvThreads) {
      y[i] = x[i];
      pv[i] = a.piv[a.voff[b] + i];
    }
    stage(d);
    __syncthreads();
    if (warp == 0) {
      // the row swaps in order, the steps that swap nothing skipped
      for (int i0 = 0; i0 < n; i0 += 32) {
        const int p = i0 + lane < n ? pv[i0 + lane] : i0 + lane;
        unsigned moves = __ballot_sync(0xffffffffu, p != i0 + lane);
        while (moves) {
          const int q = __ffs(moves) - 1;
          moves &= moves - 1;
          const int to = __shfl_sync(0xffffffffu, p, q);
          if (lane == 0) {
            const double s = y[i0 + q];
            y[i0 + q] = y[to];
            y[to] = s;
          }
        }
      }
      __syncwarp();
    }
    for (int kb = 0; kb < nblk; ++kb) {  // forward, unit lower
      const int k0 = kb * kSvB, kw = min(kSvB, n - k0);
      if (warp == 0) {
        double v = lane < kw ? y[k0 + lane] : 0.0;
#pragma unroll 8
        for (int j = 0; j < kw; ++j) {
          const double xj = __shfl_sync(0xffffffffu, v, j);
          if (lane > j) v = fma(-T[lane * kSvTS + j], xj, v);
        }
        if (lane < kw) y[k0 + lane] = v;
      }
      if (kb + 1 < nblk) fetch(k0 + kSvB, d);
      __syncthreads();
      if (kb + 1 < nblk) {
        stage(d);
        update(k0, kw, k0 + kw, n);
        __syncthreads();
      }
    }
    for (int kb = nblk - 1; kb >= 0; --kb) {  // backward; the last block's triangle is staged already
      const int k0 = kb * kSvB, kw = min(kSvB, n - k0);
      if (warp == 0) {
        double v = lane < kw ? y[k0 + lane] : 0.0;
        // v / dg by the reciprocal and one residual correction (Markstein);
        // diagonals near the ends of the range divide instead
        const double dg = lane < kw ? T[lane * kSvTS + lane] : 1.0;
        const bool plain = fabs(dg) >= 1e-290 && fabs(dg) <= 1e290;
        const double rd = 1.0 / dg;
#pragma unroll 4
        for (int j = kw - 1; j >= 0; --j) {
          const double q = v * rd;
          double xj = fma(fma(-q, dg, v), rd, q);
          if (!(plain && fabs(q) <= 1e290)) xj = v / dg;
          xj = __shfl_sync(0xffffffffu, xj, j);
          if (lane == j) v = xj;
          if (lane < j) v = fma(-T[lane * kSvTS + j], xj, v);
        }
        if (lane < kw) y[k0 + lane] = v;
      }
      if (kb > 0) fetch(k0 - kSvB, d);
      __syncthreads();
      if (kb > 0) {
        stage(d);
        update(k0, kw, 0, k0);
        __syncthreads();
      }
    }
    for (int i = tid; i < n; i += kSvThreads) x[i] = y[i];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&a.queue[1], 1u) == gridDim.x - 1) {
      a.queue[0] = 0u;
      a.queue[1] = 0u;
    }
  }
}

// A warp per system, a dot product and five shuffles per unknown: slower than
// the blocks above for one system (92 against 40 us at 64 rows), but an SM holds
// 48 or 64 systems instead of 16 CTAs whose other warps wait for the one with the
// triangle, and a small system has no 32 unknowns to fill a block with (see
// solve_by_warps).
constexpr int kSolveWarps = 8;

__global__ void __launch_bounds__(kSolveWarps * 32) batched_lu_solve_warp_kernel(const LuSolveArgs a) {
  extern __shared__ __align__(16) double sv_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double *y = sv_smem + static_cast<size_t>(warp) * a.max_n;
  while (true) {
    int item = 0;
    if (lane == 0) item = static_cast<int>(atomicAdd(&a.queue[0], 1u));
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= a.count) break;
    const int b = a.order ? a.order[item] : item;
    const int n = a.sizes[b];
    const double *L = a.LU + a.moff[b];
    const int32_t *pv = a.piv + a.voff[b];
    double *x = a.x + a.voff[b];
    for (int i = lane; i < n; i += 32) y[i] = x[i];
    __syncwarp();
    if (lane == 0) {
      for (int i = 0; i < n; ++i) {
        const int p = pv[i];
        if (p != i) { const double t = y[i]; y[i] = y[p]; y[p] = t; }
      }
    }
    __syncwarp();
    for (int i = 1; i < n; ++i) {  // forward, unit lower
      const double *row = L + static_cast<int64_t>(i) * n;
      double s = 0.0;
      for (int j = lane; j < i; j += 32) s = fma(row[j], y[j], s);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
      if (lane == 0) y[i] -= s;
      __syncwarp();
    }
    for (int i = n - 1; i >= 0; --i) {  // backward, upper with diagonal
      const double *row = L + static_cast<int64_t>(i) * n;
      double s = 0.0;
      for (int j = i + 1 + lane; j < n; j += 32) s = fma(row[j], y[j], s);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
      if (lane == 0) y[i] = (y[i] - s) / row[i];
      __syncwarp();
    }
    for (int i = lane; i < n; i += 32) x[i] = y[i];
    __syncwarp();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&a.queue[1], 1u) == gridDim.x - 1) {
      a.queue[0] = 0u;
      a.queue[1] = 0u;
    }
  }
}

// Whether a batch takes a warp per system: where its systems fill enough of the
// warps resident at once (`resident`).  A batch costs the CTAs about 0.5 ns a row
// and system, the warps 1.9 to 2.7 us a row and wave; of blocks with fewer than 32
// rows, or with few in their last 32, the CTAs gain less.  CTAs and warps, us:
// 8 rows, 1000 systems 16 and 16, 1500 20 and 16; 16 rows, 1000 22 and 25, 2000 31
// and 27, 50000 580 and 207; 40 rows, 2000 49 and 55, 3000 74 and 61, 10000 221 and
// 147; 32 rows, 3000 45 and 49, 5000 66 and 59; 72 rows, 3000 135 and 154, 5000 193
// and 172; 64 rows, 5000 147 and 147, 8000 (two waves) 227 and 265, 12000 336 and
// 285; 128 rows, 2000 141 and 307, 5000 317 and 340, 8000 500 and 635, 12000 741 and
// 670.  Larger blocks stay with the CTAs (256 rows, 3000: 547 and 777).
static bool solve_by_warps(int count, int max_n, int resident) {
  if (max_n > 160 || resident < 1) return false;
  const int64_t waves = (static_cast<int64_t>(count) + resident - 1) / resident;
  const int64_t enough = max_n <= 12                   ? 1000
                         : max_n < 32                  ? 1500
                         : max_n < 64 && max_n != 32   ? 2500
                         : max_n < 96 && max_n != 64   ? 4000
                                                       : 5000;
  return count > enough * waves;
}

static int pick_nb(int max_n) {
  if (max_n <= 640) return 32;
  if (max_n <= 1280) return 16;
  if (max_n <= 2560) return 8;
  return 0;
}

static size_t factor_smem(int nb, int max_n) {
  return (static_cast<size_t>(max_n) * nb + static_cast<size_t>(nb) * kChunk) * sizeof(double);
}

// Raises a kernel's dynamic shared-memory limit to the opt-in maximum once
// per device (a host-side attribute, so later launches and stream captures
// need no further runtime calls).
template <typename K>
static int allow_max_smem(K kernel, bool (&done)[64]) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return F3D_ERR_CUDA;
  if (done[dev]) return F3D_OK;
  int optin = 0;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return F3D_ERR_CUDA;
  // the opt-in limit covers static plus dynamic shared memory
  cudaFuncAttributes fa;
  if (cudaFuncGetAttributes(&fa, kernel) != cudaSuccess) return F3D_ERR_CUDA;
  const int dyn = optin - static_cast<int>(fa.sharedSizeBytes);
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess)
    return F3D_ERR_CUDA;
  done[dev] = true;
  return F3D_OK;
}

template <int NB>
static int launch_factor(const LuArgs &a, int max_n, cudaStream_t st) {
  const size_t smem = factor_smem(NB, max_n);
  auto k = batched_lu_factor_kernel<NB>;
  static bool done[64] = {false};
  if (allow_max_smem(k, done)) return F3D_ERR_CUDA;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kLuThreads, smem) != cudaSuccess ||
      per_sm < 1)
    per_sm = 1;
  const int grid = std::max(1, std::min(a.count, per_sm * sm_count()));
  k<<<grid, kLuThreads, smem, st>>>(a);
  return launch_status();
}

static int launch_factor_tc(const LuArgs &a, int max_n, cudaStream_t st) {
  const size_t smem = lt_smem(max_n);
  static bool done[64] = {false};
  if (allow_max_smem(lu_tc_kernel, done)) return F3D_ERR_CUDA;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, lu_tc_kernel, kLtThreads, smem) != cudaSuccess ||
      per_sm < 1)
    per_sm = 1;
  lu_tc_kernel<<<std::max(1, std::min(a.count, per_sm * sm_count())), kLtThreads, smem, st>>>(a, max_n);
  return launch_status();
}

}  // namespace f3d

extern "C" {

int f3d_batched_lu_workspace_bytes(size_t *bytes) {
  if (!bytes) return F3D_ERR_NULL;
  *bytes = 256;  // two queue counters
  return F3D_OK;
}

int f3d_batched_lu_factor_panel(double *A, const int64_t *matrix_offsets,
                                const int64_t *vector_offsets, const int32_t *sizes,
                                const int32_t *order, int32_t count, int32_t max_n, int32_t panel,
                                int32_t *piv, int32_t *info, void *workspace,
                                size_t workspace_bytes, void *stream) {
  if (count < 0 || max_n < 0) return F3D_ERR_SHAPE;
  if (count == 0) return F3D_OK;
  if (!A || !matrix_offsets || !vector_offsets || !sizes || !piv || !info) return F3D_ERR_NULL;
  if (!workspace || workspace_bytes < 256) return F3D_ERR_WORKSPACE;
  if (!f3d::aligned(A, 8)) return F3D_ERR_ALIGN;
  if (panel != 0 && panel != 8 && panel != 16 && panel != 32) return F3D_ERR_ARG;
  const int nb = panel ? panel : f3d::pick_nb(max_n);
  if (nb == 0 || f3d::factor_smem(nb, max_n) > 220 * 1024) return F3D_ERR_TOO_LARGE;
  f3d::LuArgs a{A, matrix_offsets, vector_offsets, sizes, order, piv, info,
                static_cast<unsigned *>(workspace), count};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // the tensor-core kernel takes every batch that fits its one row per thread
  // (factors measured beside the kernel: 1.7 to 4 times faster than any panel
  // width of the other at 64-256 rows); larger blocks, and an explicit panel
  // width, take the other
  if (panel == 0 && max_n <= f3d::kLtMax) return f3d::launch_factor_tc(a, max_n, st);
  if (nb == 32) return f3d::launch_factor<32>(a, max_n, st);
  if (nb == 16) return f3d::launch_factor<16>(a, max_n, st);
  return f3d::launch_factor<8>(a, max_n, st);
}

int f3d_batched_lu_factor(double *A, const int64_t *matrix_offsets, const int64_t *vector_offsets,
                          const int32_t *sizes, const int32_t *order, int32_t count, int32_t max_n,
                          int32_t *piv, int32_t *info, void *workspace, size_t workspace_bytes,
                          void *stream) {
  return f3d_batched_lu_factor_panel(A, matrix_offsets, vector_offsets, sizes, order, count, max_n, 0,
                                     piv, info, workspace, workspace_bytes, stream);
}

int f3d_batched_lu_solve(const double *LU, const int64_t *matrix_offsets,
                         const int64_t *vector_offsets, const int32_t *sizes, const int32_t *order,
                         int32_t count, int32_t max_n, const int32_t *piv, double *x,
                         void *workspace, size_t workspace_bytes, void *stream) {
  if (count < 0 || max_n < 0) return F3D_ERR_SHAPE;
  if (count == 0) return F3D_OK;
  if (!LU || !matrix_offsets || !vector_offsets || !sizes || !piv || !x) return F3D_ERR_NULL;
  if (!workspace || workspace_bytes < 256) return F3D_ERR_WORKSPACE;
  // the limit of the blocks this call takes
  const size_t warp_smem = f3d::kSolveWarps * static_cast<size_t>(max_n) * sizeof(double);
  if (warp_smem > 200 * 1024) return F3D_ERR_TOO_LARGE;
  // queue counters live after the factor's two words
  f3d::LuSolveArgs a{LU, matrix_offsets, vector_offsets, sizes, order, piv, x,
                     static_cast<unsigned *>(workspace) + 2, count, max_n};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (count > 1000 && max_n <= 160) {
    auto k = f3d::batched_lu_solve_warp_kernel;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, f3d::kSolveWarps * 32, warp_smem) != cudaSuccess)
      return F3D_ERR_CUDA;
    const int ctas = per_sm * f3d::sm_count();
    if (f3d::solve_by_warps(count, max_n, f3d::kSolveWarps * ctas)) {
      const int grid = std::min((count + f3d::kSolveWarps - 1) / f3d::kSolveWarps, ctas);
      k<<<grid, f3d::kSolveWarps * 32, warp_smem, st>>>(a);
      return f3d::launch_status();
    }
  }
  const size_t smem = (static_cast<size_t>((max_n + 1) / 2 * 2) + f3d::kSvB * f3d::kSvTS + 1) * sizeof(double) +
                      static_cast<size_t>(max_n) * sizeof(int32_t);
  auto k = f3d::batched_lu_solve_kernel;
  static bool done[64] = {false};
  if (f3d::allow_max_smem(k, done)) return F3D_ERR_CUDA;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, f3d::kSvThreads, smem) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  const int grid = std::max(1, std::min(count, per_sm * f3d::sm_count()));
  k<<<grid, f3d::kSvThreads, smem, st>>>(a);
  return f3d::launch_status();
}

}  // extern "C"
