// Batched explicit inverses of small dense FP64 blocks, and the batched
// block-diagonal matrix-vector product that applies them.
//
// fiber3d's block-diagonal preconditioner (P_inv, tstep/tstep.py:950-994)
// factors every fiber block with scipy.linalg.lu_factor
// (tstep/tstep_utils.py:1405-1419) and applies lu_solve once per GMRES
// iteration.  A substitution is a chain of 2n dependent steps; a product
// with the explicit inverse is one streaming pass over the block, so for the
// fiber blocks (4N <= 128) this file forms P_b^-1 once per time step and
// applies it as a block GEMV.  The preconditioner is the same linear
// operator as fiber3d's (to rounding); only how it is evaluated changes.
//
// Inverse: Gauss-Jordan with partial (row) pivoting, in place.  Step k picks
// a row p >= k of (to 2^-20) largest |a_pk|, swaps rows k and p, and pivots
// on (k, k):
//   a_kk <- 1/a_kk,  a_kj <- a_kj / a_kk,  a_ik <- -a_ik / a_kk,
//   a_ij <- a_ij - a_ik a_kj / a_kk      (i != k, j != k, old values).
// After n steps the array holds (PA)^-1; swapping columns k and p_k for
// k = n-1 .. 0 gives A^-1.
//
// Blocks of up to 32 rows (batched_inverse_kernel<32>): one CTA per block
// holds the whole NMAX x NMAX matrix in registers, thread t an 8 x 4 tile
// (rows 8*(t/(NMAX/4)) .., columns 4*(t%(NMAX/4)) ..), so a warp covers
// whole rows.  Per step the owners of column k publish it to
// shared memory (the pivot search is then done redundantly by every warp, no
// extra barrier), the owners of rows k and p publish those rows, and every
// thread applies the rank-1 sweep to its tile: two barriers per step.
// Blocks smaller than NMAX are padded with the identity, which the sweeps
// leave untouched.  Blocks of 33..128 rows take the blocked form
// (batched_inverse_tc_kernel): 16-column panels, no row exchanges, and the
// rank-16 updates on the FP64 tensor cores.
#include <algorithm>
#include <climits>

#include "f3d_common.cuh"

namespace f3d {

constexpr int kInvTR = 8;  // tile rows per thread
constexpr int kInvTC = 4;  // tile columns per thread

template <int NMAX>
struct InvShape {
  static constexpr int kColTiles = NMAX / kInvTC;
  static constexpr int kRowTiles = NMAX / kInvTR;
  static constexpr int kThreads = kColTiles * kRowTiles;
};

// Step k = kb + M of the Gauss-Jordan sweep on the register tiles.
// Column k is published to shared memory and zeroed in the tiles; the pivot
// row is read back with its column-k entry taken as 1, so that one update
//   a_ij <- a_ij - (c_i / pv) u_j
// gives every entry: a_kj = u_j / pv on the pivot row (which is overwritten),
// a_ik = -c_i / pv in column k, and the elimination elsewhere.
template <int NMAX, int M>
__device__ __forceinline__ void inverse_step(double (&a)[kInvTR][kInvTC], int kb, int n, int r0,
                                             int c0, int ct, int rt, int lane, int tid,
                                             double (*s_col)[NMAX], double (*s_row)[2][NMAX],
                                             int *s_piv, int &first_zero) {
  constexpr int II = M % kInvTR;  // tile row of row k in its owner
  constexpr int JJ = M % kInvTC;  // tile column of column k in its owner
  const int k = kb + M;
  if (k >= NMAX) return;
  const int par = k & 1;
  // (a) publish column k, zero it in the tiles
  if (ct == k / kInvTC) {
#pragma unroll
    for (int i = 0; i < kInvTR; ++i) {
      s_col[par][r0 + i] = a[i][JJ];
      a[i][JJ] = 0.0;
    }
  }
  __syncthreads();
  // (b) pivot, found by every warp: the first row p >= k whose magnitude
  // has the largest leading 32 bits (sign, exponent, 20 mantissa bits), i.e.
  // a pivot within a factor 1 - 2^-20 of the column maximum -- threshold
  // partial pivoting, as stable as the exact maximum.  Two warp reductions.
  unsigned key = 0u, row = 0xFFFFFFFFu;
#pragma unroll
  for (int q = 0; q < NMAX / 32; ++q) {
    const int r = lane + 32 * q;
    if (r >= k && r < n) {
      const unsigned kq =
          static_cast<unsigned>(static_cast<unsigned long long>(__double_as_longlong(fabs(s_col[par][r]))) >> 32);
      if (row == 0xFFFFFFFFu || kq > key) { key = kq; row = static_cast<unsigned>(r); }
    }
  }
  const unsigned kmax = __reduce_max_sync(0xffffffffu, row != 0xFFFFFFFFu ? key : 0u);
  const unsigned pmin = __reduce_min_sync(0xffffffffu, (row != 0xFFFFFFFFu && key == kmax) ? row : 0xFFFFFFFFu);
  const int p = pmin < static_cast<unsigned>(n) ? static_cast<int>(pmin) : k;
  // (c) publish rows k and p (column k already zero); 16-byte stores
  if (rt == k / kInvTR) {
    double2 *dst = reinterpret_cast<double2 *>(&s_row[par][0][c0]);
    dst[0] = make_double2(a[II][0], a[II][1]);
    dst[1] = make_double2(a[II][2], a[II][3]);
  }
  if (rt == p / kInvTR) {
    const int ip = p % kInvTR;
    double v[kInvTC];
#pragma unroll
    for (int j = 0; j < kInvTC; ++j) {
      v[j] = a[0][j];
#pragma unroll
      for (int i = 1; i < kInvTR; ++i) v[j] = (ip == i) ? a[i][j] : v[j];
    }
    double2 *dst = reinterpret_cast<double2 *>(&s_row[par][1][c0]);
    dst[0] = make_double2(v[0], v[1]);
    dst[1] = make_double2(v[2], v[3]);
  }
  if (tid == 0) s_piv[k] = p;
  __syncthreads();
  // (d) swap rows k and p, then the update
  const double pv = s_col[par][p];
  const bool zero_pivot = !(fabs(pv) >= 2.2250738585072014e-308);  // zero, subnormal or NaN
  if (zero_pivot && first_zero == 0) first_zero = k + 1;
  const double pinv = zero_pivot ? 0.0 : reciprocal(pv);
  double u[kInvTC];
  {
    const double2 *src = reinterpret_cast<const double2 *>(&s_row[par][1][c0]);
    const double2 u01 = src[0], u23 = src[1];
    u[0] = u01.x; u[1] = u01.y; u[2] = u23.x; u[3] = u23.y;
  }
  if (ct == k / kInvTC) u[JJ] = 1.0;
  double c[kInvTR];
  {
    const double2 *src = reinterpret_cast<const double2 *>(&s_col[par][r0]);
#pragma unroll
    for (int i = 0; i < kInvTR / 2; ++i) {
      const double2 cc = src[i];
      c[2 * i] = cc.x;
      c[2 * i + 1] = cc.y;
    }
  }
#pragma unroll
  for (int i = 0; i < kInvTR; ++i) {
    const int r = r0 + i;
    if (r == k) {
#pragma unroll
      for (int j = 0; j < kInvTC; ++j) a[i][j] = u[j] * pinv;
    } else {
      double ci;
      if (r == p) {
        const double2 *src = reinterpret_cast<const double2 *>(&s_row[par][0][c0]);
        const double2 w01 = src[0], w23 = src[1];
        a[i][0] = w01.x; a[i][1] = w01.y; a[i][2] = w23.x; a[i][3] = w23.y;
        ci = s_col[par][k];
      } else {
        ci = c[i];
      }
      const double f = ci * pinv;
#pragma unroll
      for (int j = 0; j < kInvTC; ++j) a[i][j] = fma(-f, u[j], a[i][j]);
    }
  }
}

template <int NMAX>
__global__ void __launch_bounds__(InvShape<NMAX>::kThreads, 1)
    batched_inverse_kernel(double *__restrict__ A, const int64_t *__restrict__ moff,
                           const int32_t *__restrict__ sizes, int count, float *__restrict__ A32,
                           int32_t *__restrict__ info) {
  using S = InvShape<NMAX>;
  __shared__ __align__(16) double s_col[2][NMAX];
  __shared__ __align__(16) double s_row[2][2][NMAX];  // [parity][0: old row k, 1: old row p][col]
  __shared__ int s_piv[NMAX];
  __shared__ int s_dest[NMAX];
  const int b = blockIdx.x;
  if (b >= count) return;
  const int n = sizes[b];
  if (n <= 0 || n > NMAX) return;
  double *M = A + moff[b];
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int ct = tid % S::kColTiles, rt = tid / S::kColTiles;
  const int c0 = ct * kInvTC, r0 = rt * kInvTR;

  double a[kInvTR][kInvTC];
#pragma unroll
  for (int i = 0; i < kInvTR; ++i) {
    const int r = r0 + i;
#pragma unroll
    for (int j = 0; j < kInvTC; ++j) {
      const int c = c0 + j;
      a[i][j] = (r < n && c < n) ? M[static_cast<int64_t>(r) * n + c] : (r == c ? 1.0 : 0.0);
    }
  }
  int first_zero = 0;
  // Steps run in groups of kInvTR so that k % kInvTR and k % kInvTC are
  // compile-time constants inside a step (no runtime register indexing).
  // Steps past n pivot on the identity padding and change nothing.
  for (int kb = 0; kb < n; kb += kInvTR) {
    inverse_step<NMAX, 0>(a, kb, n, r0, c0, ct, rt, lane, tid, s_col, s_row, s_piv, first_zero);
    inverse_step<NMAX, 1>(a, kb, n, r0, c0, ct, rt, lane, tid, s_col, s_row, s_piv, first_zero);
    inverse_step<NMAX, 2>(a, kb, n, r0, c0, ct, rt, lane, tid, s_col, s_row, s_piv, first_zero);
    inverse_step<NMAX, 3>(a, kb, n, r0, c0, ct, rt, lane, tid, s_col, s_row, s_piv, first_zero);
    inverse_step<NMAX, 4>(a, kb, n, r0, c0, ct, rt, lane, tid, s_col, s_row, s_piv, first_zero);
    inverse_step<NMAX, 5>(a, kb, n, r0, c0, ct, rt, lane, tid, s_col, s_row, s_piv, first_zero);
    inverse_step<NMAX, 6>(a, kb, n, r0, c0, ct, rt, lane, tid, s_col, s_row, s_piv, first_zero);
    inverse_step<NMAX, 7>(a, kb, n, r0, c0, ct, rt, lane, tid, s_col, s_row, s_piv, first_zero);
  }
  // column unscramble: X P, swaps (k, p_k) for k = n-1 .. 0
  __syncthreads();
  if (tid == 0) {
    for (int j = 0; j < n; ++j) s_dest[j] = j;  // s_dest[j] = source column of final column j
    for (int k = n - 1; k >= 0; --k) {
      const int p = s_piv[k];
      const int t = s_dest[k];
      s_dest[k] = s_dest[p];
      s_dest[p] = t;
    }
    // invert: final position of source column c
    for (int j = 0; j < n; ++j) s_piv[s_dest[j]] = j;
    info[b] = first_zero;
  }
  __syncthreads();
  float *M32 = A32 ? A32 + moff[b] : nullptr;
#pragma unroll
  for (int i = 0; i < kInvTR; ++i) {
    const int r = r0 + i;
    if (r >= n) continue;
#pragma unroll
    for (int j = 0; j < kInvTC; ++j) {
      const int c = c0 + j;
      if (c >= n) continue;
      const int64_t o = static_cast<int64_t>(r) * n + s_piv[c];
      M[o] = a[i][j];
      if (M32) M32[o] = static_cast<float>(a[i][j]);
    }
  }
}

// Blocked Gauss-Jordan for blocks of 33..128 rows (NMAX 64, 96 or 128): one CTA
// per block, the block in shared memory (padded with the identity), 16
// pivots per panel.
//  * Panel: four sub-panels of 4 columns.  NMAX threads, one row each with
//    the row's 4 entries in registers, run the 4 sweeps; the panel's other 12
//    columns then move by W R of the sub-panel, one m16n8k4 step per 16 x 8
//    tile.  (The chain of pivots bounds the kernel, and with all 16 columns
//    in registers a step is bound by the shared-memory pipe: each warp's best
//    row is posted and the pivot row read back 16 bytes at a time, about five
//    cycles an access and warp.)  Partial pivoting: the pivot of step k is a
//    row whose |a_ik|, cut to its leading 16 mantissa bits, is largest among the
//    rows not yet pivoted (a pivot within 2^-16 of the column maximum; among
//    equals the first lane, then the first warp).  The key (exponent, those bits,
//    the lane: 32 bits) makes the search one warp max-reduction and a max over
//    the warps; each warp's winner posts its row, key and reciprocal, so a step
//    needs one barrier (posts double buffered by step parity).  (12 bits: 249
//    us for 512 blocks of 128; the row posted beside its pivot instead of read
//    from the key: 265.)  Rows are never exchanged: the pivot rows are recorded
//    instead (perm).
//  * Update: every other column moves by W R (W the panel after its sweeps,
//    R the old entries of the panel's 16 pivot rows), the pivot rows
//    themselves starting from zero: one m16n8k16 step on the FP64 tensor
//    cores per 16 x 8 tile.  At 128 rows (189 KB: one block per SM) the next
//    panel's columns come first, by all warps, then the rest by half of them
//    while the others sweep that panel; up to 96 rows two blocks share an SM
//    and up to 64 rows four, which overlap by themselves.
// 512 blocks: 253 us at 128 rows, 118 at 96, 43 at 64, against 307, 286 (by the
// 128-row kernel) and 71 us with 16-column sweeps in registers and the update
// after them; one block of 128: 62 us, 78 before.  (The block in global memory
// with four CTAs per SM: 266 us.)
// Sweeping pivot (perm[k], k) for every k leaves X with X[perm[k], j] =
// (PA)^-1 (k, j), so A^-1 (k, perm[j]) = X[perm[k], j].
template <int NMAX>
struct TcInv {
  static constexpr int kS = NMAX + 4;  // block row stride (doubles): B-fragment reads 4t + g apart
  static constexpr int kWS = 20;       // W panel row stride: A-fragment reads 4g + t apart
  static constexpr int kPanels = NMAX / 16;
  static constexpr int kThreads = 256;
  static constexpr bool kAhead = NMAX > 96;      // sweep the next panel beside the update: one block per SM
  static constexpr int kW = kAhead ? 2 : 1;      // W panels held
  static constexpr size_t kSmem =
      (static_cast<size_t>(NMAX) * kS + kW * static_cast<size_t>(NMAX) * kWS + 16 * static_cast<size_t>(kS)) *
      sizeof(double);
};

template <int NMAX>
__global__ void __launch_bounds__(256, NMAX == 64 ? 4 : (NMAX == 96 ? 2 : 1))
    batched_inverse_tc_kernel(double *A, const int64_t *__restrict__ moff, const int32_t *__restrict__ sizes,
                              int count, float *__restrict__ A32, int32_t *__restrict__ info, const double *src,
                              int64_t src_ld) {
  using T = TcInv<NMAX>;
  constexpr int S = T::kS;
  extern __shared__ __align__(16) unsigned char tc_smem[];
  double *X = reinterpret_cast<double *>(tc_smem);  // [NMAX][S]
  double *W2 = X + NMAX * S;                         // [kW][NMAX][kWS], by panel parity
  double *Rs = W2 + T::kW * NMAX * T::kWS;           // [16][S]
  __shared__ __align__(16) unsigned s_key[2][4];
  __shared__ __align__(16) double s_cand[2][NMAX / 32][6];  // each warp's best row of the sub-panel and its
                                                            // pivot's reciprocal, by step parity
  __shared__ int s_zero;
  __shared__ int s_perm[NMAX];   // pivot row of step k
  __shared__ int s_step[NMAX];   // step whose pivot is row r (NMAX: not yet)
  const int b = blockIdx.x;
  if (b >= count) return;
  const int n = sizes[b];
  if (n <= 0 || n > NMAX) return;
  double *M = A + moff[b];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // (src: the block is read from there, row stride src_ld, instead of in place)
  const double *from = src ? src : M;
  const int64_t ldm = src ? src_ld : n;
  if (n == NMAX && (ldm & 1) == 0 && (reinterpret_cast<uintptr_t>(from) & 15) == 0) {
    for (int e = tid; e < NMAX * NMAX / 2; e += T::kThreads)
      cp_async16(&X[e / (NMAX / 2) * S + 2 * (e % (NMAX / 2))], from + e / (NMAX / 2) * ldm + 2 * (e % (NMAX / 2)));
    cp_async_commit();
    cp_async_wait<0>();
  } else {
#pragma unroll 4
    for (int e = tid; e < NMAX * NMAX; e += T::kThreads) {
      const int r = e / NMAX, c = e % NMAX;
      X[r * S + c] = (r < n && c < n) ? from[r * ldm + c] : (r == c ? 1.0 : 0.0);
    }
  }
  for (int r = tid; r < NMAX; r += T::kThreads) s_step[r] = NMAX;
  if (tid < 8) s_key[tid >> 2][tid & 3] = 0u;
  if (tid == 0) s_zero = INT_MAX;
  __syncthreads();
  int first_zero = 0;  // the first zero pivot this thread's row was (a row is a pivot once)
  // this thread's row in the pivot search; all 0 once it has been a pivot
  unsigned key_mask = 0x7ffffff0u, key_add = 63u - lane;
  constexpr int kRT = NMAX / 16, kCT = NMAX / 8, kPW = NMAX / 32;
  const int g = lane >> 2, t = lane & 3;

  // panel p (warps 0 .. kPW - 1): its sweeps, W to its buffer and to the panel's columns
  auto panel = [&](int p) {
    const int c0 = 16 * p, i = tid;
    double *Ws = W2 + (T::kAhead ? p & 1 : 0) * NMAX * T::kWS;
    auto bar = [] { asm volatile("bar.sync 1, %0;" ::"n"(NMAX) : "memory"); };
#pragma unroll
    for (int j = 0; j < 16; j += 2)
      *reinterpret_cast<double2 *>(&Ws[i * T::kWS + j]) = *reinterpret_cast<const double2 *>(&X[i * S + c0 + j]);
    for (int s0 = 0; s0 < 16; s0 += 4) {
      double v[4];
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        const double2 w = *reinterpret_cast<const double2 *>(&Ws[i * T::kWS + s0 + j]);
        v[j] = w.x;
        v[j + 1] = w.y;
      }
      int piv[4];  // the sub-panel's pivot rows
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        const int par = jj & 1, k = c0 + s0 + jj;
        // pivot key: exponent and 16 mantissa bits of |a_ik| (plus one), then the
        // lane (the first among equals): at least 32 for a row not yet pivoted,
        // else 0 (a NaN whose bits are all set wraps; see the end)
        const unsigned key = 2u * (static_cast<unsigned>(__double2hiint(v[jj])) & key_mask) + key_add;
        const double rcp = reciprocal(v[jj]);  // beside the search
        const unsigned wmax = __reduce_max_sync(0xffffffffu, key);
        if (key == wmax) {  // this warp's winner posts its row (live keys are distinct; a warp
                            // with no live row posts garbage under key 0, which never wins)
          s_key[par][warp] = wmax;
          double *const c = s_cand[par][warp];
          *reinterpret_cast<double2 *>(c) = make_double2(v[0], v[1]);
          *reinterpret_cast<double2 *>(c + 2) = make_double2(v[2], v[3]);
          c[4] = rcp;
        }
        bar();
        const uint4 h = *reinterpret_cast<const uint4 *>(s_key[par]);
        const unsigned best = max(max(h.x, h.y), max(h.z, h.w));
        const int bw = h.x == best ? 0 : (h.y == best ? 1 : (h.z == best ? 2 : 3));
        const int pr = 32 * bw + 31 - static_cast<int>(best & 31u);
        const double *prow = s_cand[par][bw];
        const double inv = prow[4];
        piv[jj] = pr;
        if (i == pr) {
          s_perm[k] = i;
          s_step[i] = k;
          key_mask = key_add = 0u;
          if (first_zero == 0 && !(fabs(v[jj]) >= 2.2250738585072014e-308)) first_zero = k + 1;
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] = (j == jj) ? inv : v[j] * inv;
        } else {
          const double l = v[jj] * inv;
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] = (j == jj) ? -l : fma(-l, prow[j], v[j]);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; j += 2)
        *reinterpret_cast<double2 *>(&Ws[i * T::kWS + s0 + j]) = make_double2(v[j], v[j + 1]);
      bar();
      // the panel's other 12 columns: one m16n8k4 step per 16 x 8 tile (four
      // tiles a warp, row tiles first), the four pivot rows taken into registers
      // before any of them changes
      const int pt = t == 0 ? piv[0] : (t == 1 ? piv[1] : (t == 2 ? piv[2] : piv[3]));
      double2 o[4][2];
      double af[4][2], b4[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int id = 4 * warp + q, rt = id % kRT, ch = 8 * (id / kRT);
        b4[q] = Ws[pt * T::kWS + ch + g];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = 16 * rt + g + 8 * h;
          const bool keep = r != piv[0] && r != piv[1] && r != piv[2] && r != piv[3];
          const double2 x = *reinterpret_cast<const double2 *>(&Ws[r * T::kWS + ch + 2 * t]);
          o[q][h] = keep ? x : make_double2(0.0, 0.0);
          af[q][h] = Ws[r * T::kWS + s0 + t];
        }
      }
      bar();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int id = 4 * warp + q, rt = id % kRT, cc = 8 * (id / kRT) + 2 * t;
        double dd[4] = {o[q][0].x, o[q][0].y, o[q][1].x, o[q][1].y};
        mma_f64_1684(dd, af[q][0], af[q][1], b4[q]);
        if ((cc & ~3) != s0) {  // (the sub-panel's own columns hold its W)
          double *x = &Ws[(16 * rt + g) * T::kWS + cc];
          *reinterpret_cast<double2 *>(x) = make_double2(dd[0], dd[1]);
          *reinterpret_cast<double2 *>(x + 8 * T::kWS) = make_double2(dd[2], dd[3]);
        }
      }
      bar();
    }
#pragma unroll
    for (int j = 0; j < 16; j += 2)
      *reinterpret_cast<double2 *>(&X[i * S + c0 + j]) = *reinterpret_cast<const double2 *>(&Ws[i * T::kWS + j]);
  };
  // panel p's update of row tile rt, column tiles ct = ct0, ct0 + step, ...
  // outside the panels p and `skip`: X <- [row not a pivot of this panel] X + W R
  auto update = [&](int p, int skip, int rt, int ct0, int ct1, int step) {
    const double *Ws = W2 + (T::kAhead ? p & 1 : 0) * NMAX * T::kWS;
    const int r0 = 16 * rt + g, r1 = r0 + 8;
    double af[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) af[q] = Ws[(r0 + 8 * (q & 1)) * T::kWS + t + 4 * (q >> 1)];
    const bool keep0 = (s_step[r0] >> 4) != p, keep1 = (s_step[r1] >> 4) != p;
    for (int ct = ct0; ct < ct1; ct += step) {
      if ((ct >> 1) == p || (ct >> 1) == skip) continue;
      const int c = 8 * ct;
      double bf[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) bf[j] = Rs[(t + 4 * j) * S + c + g];
      double2 *x0 = reinterpret_cast<double2 *>(X + r0 * S + c + 2 * t);
      double2 *x1 = reinterpret_cast<double2 *>(X + r1 * S + c + 2 * t);
      const double2 o0 = *x0, o1 = *x1;
      double dd[4] = {keep0 ? o0.x : 0.0, keep0 ? o0.y : 0.0, keep1 ? o1.x : 0.0, keep1 ? o1.y : 0.0};
      mma_f64_16816(dd, af, bf);
      *x0 = make_double2(dd[0], dd[1]);
      *x1 = make_double2(dd[2], dd[3]);
    }
  };

  auto all_but = [&](int p, int skip, int w0) {  // warps w0 .. 7: column tiles of one parity each
    for (int it = warp - w0; it < 2 * kRT; it += 8 - w0) update(p, skip, it >> 1, it & 1, kCT, 2);
  };

  if (warp < kPW) panel(0);
  for (int p = 0; p < T::kPanels; ++p) {
    __syncthreads();
    // the panel's pivot rows as they were before the panel (outside its columns)
    for (int e = tid; e < 16 * NMAX / 2; e += T::kThreads) {
      const int jj = e / (NMAX / 2), c = 2 * (e % (NMAX / 2));
      if ((c >> 4) != p)
        *reinterpret_cast<double2 *>(&Rs[jj * S + c]) =
            *reinterpret_cast<const double2 *>(&X[s_perm[16 * p + jj] * S + c]);
    }
    __syncthreads();
    if (T::kAhead && p + 1 < T::kPanels) {
      // the next panel's columns first, so that its sweeps run beside the rest
      if (warp < kRT) update(p, -1, warp, 2 * (p + 1), 2 * (p + 2), 1);
      __syncthreads();
      if (warp < kPW)
        panel(p + 1);
      else
        all_but(p, p + 1, kPW);
    } else {
      all_but(p, -1, 0);
      if (p + 1 < T::kPanels) {
        __syncthreads();
        if (warp < kPW) panel(p + 1);
      }
    }
  }
  __syncthreads();
  // A^-1 (k, c) = X[perm[k], step[c]]: coalesced stores of the block's rows (a row
  // that a wrapped key kept from being a pivot reads its padding, column NMAX)
  float *M32 = A32 ? A32 + moff[b] : nullptr;
  for (int e = tid; e < n * n; e += T::kThreads) {
    const int k = e / n, c = e % n;
    const double v = X[s_perm[k] * S + s_step[c]];
    M[e] = v;
    if (M32) M32[e] = static_cast<float>(v);
  }
  // the first step whose pivot was zero, over the threads that held pivots
  if (first_zero) atomicMin(&s_zero, first_zero);
  __syncthreads();
  if (tid == 0) info[b] = s_zero == INT_MAX ? 0 : s_zero;
}

// y_b = M_b x_b for every block b (M row-major n_b x n_b at moff[b], x and y
// at voff[b]), a CTA per block, 8 lanes per row, FP64 accumulation.  FP64: ROWS
// rows 16 apart and U loads a row (16 bytes each where the block is aligned) in
// flight per lane.  Bound by HBM, or by L2 where the blocks stay there, so what
// counts is the bytes in flight and, in L2, the instructions beside them; the
// registers hold both down for small blocks.  1 x 4 up to 16 rows (ROWS x U), 2 x
// 2 up to 32, 4 x 2 up to 96, 4 x 4 above.  From L2 / from HBM, us, against one
// load at a time and against rows streamed through cp.async rings: 600 blocks of
// 128 rows 12 / 25 (27 / 43, 22 / 27), 2000 of 128 47 / 57 (74 / 86, 50 / 61), 600
// of 96 10 / 18 (12 / 24, 17 / 20), 2000 of 64 12 / 20 (13 / 25, 21 / 25), 10000 of
// 32 18 / 27 (20 / 31, 42 / 47), 50000 of 8 33 / 47 (35 / 55, 72 / 96), one of 1000
// 127 / 250 (521 / 1540, 253 / 283).
template <int ROWS, int U>
__global__ void __launch_bounds__(128) block_gemv_kernel(const double *__restrict__ M,
                                                         const int64_t *__restrict__ moff,
                                                         const int64_t *__restrict__ voff,
                                                         const int32_t *__restrict__ sizes, int count,
                                                         const double *__restrict__ x, double *__restrict__ y) {
  extern __shared__ __align__(16) double xs[];
  const int b = blockIdx.x;
  if (b >= count) return;
  const int n = sizes[b];
  const double *Mb = M + moff[b], *xb = x + voff[b];
  double *yb = y + voff[b];
  for (int i = threadIdx.x; i < n; i += blockDim.x) xs[i] = xb[i];
  __syncthreads();
  const bool vec = ((reinterpret_cast<uintptr_t>(Mb) & 15) == 0) && (n % 2 == 0);
  const int sub = threadIdx.x & 7, grp = threadIdx.x >> 3;  // lane within the row group, 16 row groups
  for (int r0 = 0; r0 < n; r0 += 16 * ROWS) {
    const int r = r0 + grp;
    double s[ROWS];
#pragma unroll
    for (int q = 0; q < ROWS; ++q) s[q] = 0.0;
    if (vec) {
      for (int c0 = 2 * sub; c0 < n; c0 += 16 * U) {
        double2 v[ROWS][U];
#pragma unroll
        for (int q = 0; q < ROWS; ++q)
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int c = c0 + 16 * u;
            v[q][u] = make_double2(0.0, 0.0);
            if (c < n && r + 16 * q < n)
              v[q][u] = *reinterpret_cast<const double2 *>(Mb + static_cast<int64_t>(r + 16 * q) * n + c);
          }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int c = c0 + 16 * u;
          if (c < n) {
            const double2 w = *reinterpret_cast<const double2 *>(xs + c);
#pragma unroll
            for (int q = 0; q < ROWS; ++q) s[q] = fma(v[q][u].y, w.y, fma(v[q][u].x, w.x, s[q]));
          }
        }
      }
    } else {
      for (int c0 = sub; c0 < n; c0 += 8 * U) {
        double v[ROWS][U];
#pragma unroll
        for (int q = 0; q < ROWS; ++q)
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int c = c0 + 8 * u;
            v[q][u] = c < n && r + 16 * q < n ? Mb[static_cast<int64_t>(r + 16 * q) * n + c] : 0.0;
          }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int c = c0 + 8 * u;
          if (c < n) {
#pragma unroll
            for (int q = 0; q < ROWS; ++q) s[q] = fma(v[q][u], xs[c], s[q]);
          }
        }
      }
    }
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
#pragma unroll
      for (int off = 1; off < 8; off <<= 1) s[q] += __shfl_xor_sync(0xffffffffu, s[q], off);
      if (sub == 0 && r + 16 * q < n) yb[r + 16 * q] = s[q];
    }
  }
}

// The FP32 copy: one row and one load (16 bytes where the block is aligned) at a
// time per lane, FP64 accumulation.
__global__ void __launch_bounds__(128) block_gemv_f32_kernel(const float *__restrict__ M,
                                                             const int64_t *__restrict__ moff,
                                                             const int64_t *__restrict__ voff,
                                                             const int32_t *__restrict__ sizes,
                                                             int count, const double *__restrict__ x,
                                                             double *__restrict__ y) {
  extern __shared__ __align__(16) double xs[];
  const int b = blockIdx.x;
  if (b >= count) return;
  const int n = sizes[b];
  const float *Mb = M + moff[b];
  const double *xb = x + voff[b];
  for (int i = threadIdx.x; i < n; i += blockDim.x) xs[i] = xb[i];
  __syncthreads();
  const bool vec = ((reinterpret_cast<uintptr_t>(Mb) & 15) == 0) && (n % 4 == 0);
  const int sub = threadIdx.x & 7;          // lane within the row group
  const int grp = threadIdx.x >> 3;         // 16 row groups per CTA
  for (int r = grp; r < n; r += 16) {
    const float *row = Mb + static_cast<int64_t>(r) * n;
    double s = 0.0;
    if (vec) {
      for (int c = sub * 4; c < n; c += 32) {
        const float4 v = *reinterpret_cast<const float4 *>(row + c);
        s = fma(static_cast<double>(v.x), xs[c], s);
        s = fma(static_cast<double>(v.y), xs[c + 1], s);
        s = fma(static_cast<double>(v.z), xs[c + 2], s);
        s = fma(static_cast<double>(v.w), xs[c + 3], s);
      }
    } else {
      for (int c = sub; c < n; c += 8) s = fma(static_cast<double>(row[c]), xs[c], s);
    }
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    if (sub == 0) y[voff[b] + r] = s;
  }
}

}  // namespace f3d

namespace f3d {
// Q (128 x 128, packed) = inverse of the 128 x 128 block at src, row stride
// ld; off = {0} and size = {128} on the device.
int pivot_block_inverse(const double *src, int64_t ld, double *Q, const int64_t *off, const int32_t *size,
                        int32_t *info, cudaStream_t st) {
  using T = TcInv<128>;
  if (cudaFuncSetAttribute(batched_inverse_tc_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(T::kSmem)) != cudaSuccess)
    return F3D_ERR_CUDA;
  batched_inverse_tc_kernel<128><<<1, T::kThreads, T::kSmem, st>>>(Q, off, size, 1, nullptr, info, src, ld);
  return launch_status();
}
}  // namespace f3d

extern "C" {

int f3d_batched_inverse(double *A, const int64_t *matrix_offsets, const int32_t *sizes,
                        int32_t count, int32_t max_n, float *A32, int32_t *info, void *stream) {
  if (count < 0 || max_n < 0) return F3D_ERR_SHAPE;
  if (count == 0) return F3D_OK;
  if (!A || !matrix_offsets || !sizes || !info) return F3D_ERR_NULL;
  if (max_n > 128) return F3D_ERR_TOO_LARGE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (max_n <= 32) {
    f3d::batched_inverse_kernel<32><<<count, f3d::InvShape<32>::kThreads, 0, st>>>(
        A, matrix_offsets, sizes, count, A32, info);
  } else if (max_n <= 64) {
    using T = f3d::TcInv<64>;
    if (cudaFuncSetAttribute(f3d::batched_inverse_tc_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(T::kSmem)) != cudaSuccess)
      return F3D_ERR_CUDA;
    f3d::batched_inverse_tc_kernel<64><<<count, T::kThreads, T::kSmem, st>>>(A, matrix_offsets, sizes, count, A32,
                                                                             info, nullptr, 0);
  } else if (max_n <= 96) {
    using T = f3d::TcInv<96>;
    if (cudaFuncSetAttribute(f3d::batched_inverse_tc_kernel<96>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(T::kSmem)) != cudaSuccess)
      return F3D_ERR_CUDA;
    f3d::batched_inverse_tc_kernel<96><<<count, T::kThreads, T::kSmem, st>>>(A, matrix_offsets, sizes, count, A32,
                                                                             info, nullptr, 0);
  } else {
    using T = f3d::TcInv<128>;
    if (cudaFuncSetAttribute(f3d::batched_inverse_tc_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(T::kSmem)) != cudaSuccess)
      return F3D_ERR_CUDA;
    f3d::batched_inverse_tc_kernel<128><<<count, T::kThreads, T::kSmem, st>>>(A, matrix_offsets, sizes, count,
                                                                              A32, info, nullptr, 0);
  }
  return f3d::launch_status();
}

int f3d_block_gemv(int precision, const void *M, const int64_t *matrix_offsets,
                   const int64_t *vector_offsets, const int32_t *sizes, int32_t count,
                   int32_t max_n, const double *x, double *y, void *stream) {
  if (count < 0 || max_n < 0) return F3D_ERR_SHAPE;
  if (count == 0) return F3D_OK;
  if (!M || !matrix_offsets || !vector_offsets || !sizes || !x || !y) return F3D_ERR_NULL;
  if (x == y) return F3D_ERR_ARG;
  const size_t smem = static_cast<size_t>(max_n) * sizeof(double);
  if (smem > 48 * 1024) return F3D_ERR_TOO_LARGE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (precision == F3D_FP64) {
    auto kernel = max_n <= 16 ? f3d::block_gemv_kernel<1, 4>
                  : max_n <= 32 ? f3d::block_gemv_kernel<2, 2>
                  : max_n <= 96 ? f3d::block_gemv_kernel<4, 2>
                                : f3d::block_gemv_kernel<4, 4>;
    kernel<<<count, 128, smem, st>>>(
        static_cast<const double *>(M), matrix_offsets, vector_offsets, sizes, count, x, y);
  } else if (precision == F3D_FP32C) {
    f3d::block_gemv_f32_kernel<<<count, 128, smem, st>>>(
        static_cast<const float *>(M), matrix_offsets, vector_offsets, sizes, count, x, y);
  } else {
    return F3D_ERR_ARG;
  }
  return f3d::launch_status();
}

}  // extern "C"
