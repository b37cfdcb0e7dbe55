// Rows of an FP64 matrix times a vector, streamed by independent warps.
#pragma once

#include "f3d_common.cuh"

namespace f3d {

// A warp takes its rows two at a time and streams them, 64 columns a stage with
// the same part of x, through a ring of its own in shared memory (cp.async; a
// lane reads back only what it copied, so nothing waits for another lane).
// Bound by HBM, or by L2 where the matrix stays there: what counts is the bytes
// in flight, which the rings hold without registers (144 KB per SM for one matrix).
// Loading through registers, four rows of a warp one after the other behind
// CTA-wide staging of x, drained the loads at each row and chunk: 82 us for
// 3600 x 3600, 188 us for 9000 x 9000 and 446 us for 18000 x 18000 from HBM,
// against 29, 121 and 410 us (6.3 TB/s) here; four matrices of 1206 in one launch
// 33 and 12 us.  (Four rows: the same; eight: 5 % slower at 12000; a quarter of the
// bytes in flight: 20 %.)
constexpr int kGemvRows = 2, kGemvDepth = 6;
template <int ROWS = kGemvRows, int DEPTH = kGemvDepth>
constexpr int gemv_ring_doubles() {
  return DEPTH * (ROWS + 1) * 64;  // x and the rows
}
constexpr size_t kGemvWarpSmem = gemv_ring_doubles() * sizeof(double);

__device__ __forceinline__ void gemv_copy8(double *smem, const double *gmem, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_addr(smem)), "l"(gmem), "r"(valid ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void gemv_copy16(double *smem, const double *gmem, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(smem)), "l"(gmem), "r"(valid ? 16 : 0)
               : "memory");
}

// y[r] = M[r] . x for r in [r_lo, r_hi), by one warp; ring: gemv_ring_doubles
// of its own, 16-byte aligned.  VEC 2: rows 16-byte aligned and cols even (16-byte
// copies); VEC 1: any rows.  Columns past the last count as zero times zero.
template <int VEC, int ROWS = kGemvRows, int DEPTH = kGemvDepth>
__device__ __forceinline__ void gemv_stream_rows(const double *__restrict__ M, const double *__restrict__ x,
                                                 double *y, int64_t r_lo, int64_t r_hi, int64_t cols, int64_t ld,
                                                 double *ring) {
  constexpr int kStage = (ROWS + 1) * 64;
  const int lane = threadIdx.x & 31;
  // this lane's two columns of a stage
  const int l0 = VEC == 2 ? 2 * lane : lane, l1 = VEC == 2 ? l0 + 1 : l0 + 32;
  const int64_t stages = (cols + 63) / 64;
  // the copies' place in the stream: stage ps of the rows from pr, slot pb
  int64_t pr = r_lo, ps = 0;
  int pb = 0;
  auto copy = [&]() {
    if (pr < r_hi) {
      const int64_t c0 = 64 * ps + l0, c1 = 64 * ps + l1;
      const bool v0 = c0 < cols, v1 = c1 < cols;
      double *d = ring + pb * kStage;
      gemv_copy8(d + l0, v0 ? x + c0 : x, v0);
      gemv_copy8(d + l1, v1 ? x + c1 : x, v1);
#pragma unroll
      for (int q = 0; q < ROWS; ++q) {
        const bool in = pr + q < r_hi;
        const double *row = M + (pr + q) * ld;
        if (VEC == 2) {
          gemv_copy16(d + 64 * (q + 1) + l0, v0 && in ? row + c0 : M, v0 && in);
        } else {
          gemv_copy8(d + 64 * (q + 1) + l0, v0 && in ? row + c0 : M, v0 && in);
          gemv_copy8(d + 64 * (q + 1) + l1, v1 && in ? row + c1 : M, v1 && in);
        }
      }
      if (++ps == stages) {
        ps = 0;
        pr += ROWS;
      }
      if (++pb == DEPTH) pb = 0;
    }
    cp_async_commit();
  };
#pragma unroll
  for (int d = 0; d < DEPTH - 1; ++d) copy();
  int b = 0;
  for (int64_t r = r_lo; r < r_hi; r += ROWS) {
    double acc[ROWS];
#pragma unroll
    for (int q = 0; q < ROWS; ++q) acc[q] = 0.0;
    for (int64_t s = 0; s < stages; ++s) {
      cp_async_wait<DEPTH - 2>();
      const double *d = ring + b * kStage;
      const double x0 = d[l0], x1 = d[l1];
#pragma unroll
      for (int q = 0; q < ROWS; ++q) {
        const double *m = d + 64 * (q + 1);
        acc[q] = fma(m[l1], x1, fma(m[l0], x0, acc[q]));
      }
      if (++b == DEPTH) b = 0;
      copy();  // into the slot read one stage before
    }
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
      double a = acc[q];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
      if (lane == 0 && r + q < r_hi) y[r + q] = a;
    }
  }
  cp_async_wait<0>();
}

}  // namespace f3d
