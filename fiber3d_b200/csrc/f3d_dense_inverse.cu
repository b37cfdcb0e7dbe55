// Explicit inverse of a dense FP64 matrix: the periphery operator's inverse
// that the shell preconditioner applies (fiber3d factors the dense shell
// matrix once with scipy.linalg.lu_factor, tstep/tstep.py:327-348, and
// applies lu_solve per GMRES iteration, tstep.py:950-994; here the inverse is
// formed once and applied as a GEMV), and the rigid-body blocks
// (tstep/tstep_utils.py:1341-1386).
//
// Blocked in-place Gauss-Jordan elimination ("sweep" of one 128-row block per
// step).  With b the step's block of rows/columns and r the rest, a step
// replaces
//   A_bb <- Q = A_bb^-1,   A_rb <- -A_rb Q,   A_br <- Q A_br,
//   A_rr <- A_rr - A_rb Q A_br;
// after the last step the array holds A^-1 (2 n^3 flops, as LU + inversion).
// In terms of the panel W = [-A_rb Q; Q] (the new column block) and R = A_b.
// (the old block row): every column J outside b becomes
//   A_.J <- [rows outside b] A_.J + W R_.J
// one FP64 GEMM of rank 128.  Pivoting is local: Q comes from the batched
// inverse's Gauss-Jordan kernel with partial pivoting inside the 128 x 128
// block, which reads the block where it stands (pivot_block_inverse); there
// is no row exchange across blocks.  Block
// elimination without global pivoting is stable for the operators this
// library inverts (second-kind boundary integral operators, whose diagonal
// blocks carry the 1/w-scaled identity): on spheres of 1000 and 2000 nodes
// the result agrees with an LU-with-partial-pivoting inverse to 3e-14 and
// entries grow by at most 1.06 during elimination.  A zero pivot inside a
// block is reported (F3D_ERR_SINGULAR).
//
// Per step: the pivot block is inverted (one CTA); gj_panel_kernel forms W in
// place in the panel columns and copies the old block row to R (a CTA per 32
// rows); gj_update_kernel updates every other tile; both on the FP64 tensor
// cores (mma.sync m16n8k16).  The update is persistent, two CTAs per SM (4
// warps of 32 x 64 outputs, tiles of 64 x 128), each walking its tiles with one
// continuous stream of operand chunks (32 k, cp.async, a two-stage ring, one
// barrier per chunk) across tile boundaries; a tile's old values are prefetched
// into L2 when its first chunk is requested and added in its epilogue.
#include <algorithm>
#include <vector>

#include "f3d_common.cuh"

namespace f3d {
namespace {

constexpr int kGjB = 128;             // rows/columns of a step and of a tile
// panel: 128 threads, 4 warps of 16 x 64 outputs, 32 rows per CTA; operand
// strides as the update's below
constexpr int kGpThreads = 128;
constexpr int kGpM = 32;
// update: 128 threads, 4 warps of 32 x 64 outputs on the FP64 tensor cores
// (mma.sync m16n8k16), operands in a two-stage ring of 32-k chunks.
// Shared row strides (doubles) chosen so that every fragment read is two
// conflict-free wavefronts: W chunk [64][36] (row-major A fragments: 4g + t
// distinct mod 16 over a half-warp), R chunk [32][132] (k-major B
// fragments: 4t + g).
constexpr int kGuThreads = 128;
constexpr int kGuM = 64;  // rows of an update tile (128 columns)
constexpr int kGuKC = 32, kGuChunks = kGjB / kGuKC, kGuStages = 2;
constexpr int kGuAS = 36, kGuBS = 132;
constexpr int kGuABuf = kGuM * kGuAS, kGuBBuf = kGuKC * kGuBS;
constexpr size_t kGjSmemUpdate =
    static_cast<size_t>(kGuStages) * (static_cast<size_t>(kGuABuf) + kGuBBuf) * sizeof(double);
constexpr int kGpABuf = kGpM * kGuAS;
constexpr size_t kGjSmemPanel = 2 * (static_cast<size_t>(kGpABuf) + kGuBBuf) * sizeof(double);

struct GjArgs {
  double *A;        // np x np (leading dimension ld), np a multiple of 128
  double *R;        // 128 x ld: the step's block row before the step
  const double *Q;  // 128 x 128: inverse of the step's pivot block
  int64_t ld;
  int s;            // step: pivot block index
  int *err;         // the device error word (read by the host after the last step)
};

// The panel: W_I = -A(I, b) Q for rows I outside the pivot block, W_s = Q,
// written in place into the panel columns, on the FP64 tensor cores, 32 rows
// per CTA; and the block row R as it was before the step, a 32 x 128 piece per
// CTA.  32 rows leave enough CTAs for every SM from 37 tiles on, and a quarter
// of the time of 128-row CTAs below that: 28 us a step at 10 and at 71 tiles
// for 128 rows with FP64 FMAs, 9 and 16 us now, the copy of R (3.4 and 6.6 us)
// included.
__global__ void __launch_bounds__(kGpThreads, 2) gj_panel_kernel(const GjArgs a) {
  extern __shared__ __align__(16) unsigned char gj_smem[];
  double *As = reinterpret_cast<double *>(gj_smem);  // [2][32][kGuAS]: A[row][k]
  double *Bs = As + 2 * kGpABuf;                      // [2][32][kGuBS]: Q[k][col]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int64_t row0 = static_cast<int64_t>(blockIdx.x) * kGpM, k0 = static_cast<int64_t>(a.s) * kGjB;
  // this CTA's piece of R: rows 32 (x % 4) .. + 31 of the block, column tile x / 4
  // (the panel's own columns are not read from R)
  const int J = blockIdx.x / (kGjB / kGpM), rp = kGpM * (blockIdx.x % (kGjB / kGpM));
  if (J != a.s) {
    const double *src = a.A + (k0 + rp + (tid >> 6)) * a.ld + static_cast<int64_t>(J) * kGjB + 2 * (tid & 63);
    double *dst = a.R + (rp + (tid >> 6)) * a.ld + static_cast<int64_t>(J) * kGjB + 2 * (tid & 63);
    double2 v[kGpM / 2];
#pragma unroll
    for (int i = 0; i < kGpM / 2; ++i) v[i] = *reinterpret_cast<const double2 *>(src + 2 * i * a.ld);
#pragma unroll
    for (int i = 0; i < kGpM / 2; ++i) *reinterpret_cast<double2 *>(dst + 2 * i * a.ld) = v[i];
  }
  if (row0 >= k0 && row0 < k0 + kGjB) {
    for (int i = tid; i < kGpM * kGjB / 2; i += kGpThreads) {
      const int r = i / (kGjB / 2), c2 = i % (kGjB / 2);
      reinterpret_cast<double2 *>(a.A + (row0 + r) * a.ld + k0)[c2] =
          reinterpret_cast<const double2 *>(a.Q + (row0 - k0 + r) * kGjB)[c2];
    }
    return;
  }
  auto load = [&](int c) {
    double *as = As + (c & 1) * kGpABuf, *bs = Bs + (c & 1) * kGuBBuf;
#pragma unroll
    for (int v = 0; v < kGpM / 8; ++v) {  // 32 rows x 16 segments of 16 B
      const int m = (tid >> 4) + 8 * v;
      cp_async16(as + m * kGuAS + 2 * (tid & 15), a.A + (row0 + m) * a.ld + k0 + c * kGuKC + 2 * (tid & 15));
    }
#pragma unroll
    for (int v = 0; v < kGuKC / 2; ++v) {  // 32 rows x 64 segments of 16 B
      const int kk = (tid >> 6) + 2 * v;
      cp_async16(bs + kk * kGuBS + 2 * (tid & 63), a.Q + (c * kGuKC + kk) * kGjB + 2 * (tid & 63));
    }
    cp_async_commit();
  };
  const int wr = 16 * (warp >> 1), wc = 64 * (warp & 1);
  double acc[8][4];
#pragma unroll
  for (int ni = 0; ni < 8; ++ni)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[ni][i] = 0.0;
  load(0);
  for (int c = 0; c < kGuChunks; ++c) {
    cp_async_wait<0>();
    __syncthreads();
    if (c + 1 < kGuChunks) load(c + 1);
#pragma unroll
    for (int ks = 0; ks < kGuKC / 16; ++ks) {
      const double *as = As + (c & 1) * kGpABuf + (wr + g) * kGuAS + 16 * ks + t;
      const double *bs = Bs + (c & 1) * kGuBBuf + (16 * ks + t) * kGuBS + wc + g;
      double af[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) af[i] = as[8 * (i & 1) * kGuAS + 4 * (i >> 1)];
#pragma unroll
      for (int ni = 0; ni < 8; ++ni) {
        double bf[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) bf[j] = bs[4 * j * kGuBS + 8 * ni];
        mma_f64_16816(acc[ni], af, bf);
      }
    }
  }
  // (every thread's last reads of A were the copies waited for before the last barrier)
  double *o = a.A + (row0 + wr + g) * a.ld + k0 + wc + 2 * t;
#pragma unroll
  for (int ni = 0; ni < 8; ++ni) {
    *reinterpret_cast<double2 *>(o + 8 * ni) = make_double2(-acc[ni][0], -acc[ni][1]);
    *reinterpret_cast<double2 *>(o + 8 * a.ld + 8 * ni) = make_double2(-acc[ni][2], -acc[ni][3]);
  }
}

// The update of every tile outside the panel columns, persistent: CTA x
// takes tiles x, x + gridDim.x, ... (64 rows x 128 columns, row-major over
// (I, J), J skipping the panel), its chunks one continuous stream through a
// two-stage ring across tile boundaries (one barrier per chunk: wait for chunk
// g, barrier, issue chunk g + 1 into the stage chunk g - 1 used, compute chunk
// g).  Warp w computes rows 32 (w / 2) .. + 31 and columns 64 (w % 2) .. + 63
// of the tile as 2 x 8 tensor-core tiles of 16 x 8.  A tile's old values are
// prefetched into L2 (bulk prefetch, no shared memory) when its first chunk
// is requested, and read from there in its epilogue.
//
// Two CTAs share an SM, so that one multiplies while the other is in a tile's
// epilogue (128 KB in and out of L2 after only 128 k of products) or at a
// barrier: one CTA of 8 warps per SM with tiles of 128 x 128 had the tensor
// pipe active for 66 % of the time.  All updates of a 9000-row inverse (1.46
// Tflop): 61.0 ms that way, 56.3 with two CTAs, 51.0 with the copies spread over
// the products and the epilogue's loads requested ahead (47.4 with no epilogue
// at all, 41.3 without the copies too).
__global__ void __launch_bounds__(kGuThreads, 2) gj_update_kernel(const GjArgs a, int tiles) {
  extern __shared__ __align__(16) unsigned char gj_smem[];
  double *As = reinterpret_cast<double *>(gj_smem);  // [2][64][kGuAS]: W[row][k]
  double *Bs = As + kGuStages * kGuABuf;              // [2][32][kGuBS]: R[k][col]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wr = 32 * (warp >> 1), wc = 64 * (warp & 1);
  const int ncol = tiles - 1;
  const int64_t ntile = static_cast<int64_t>(ncol) * tiles * (kGjB / kGuM);
  const int64_t first = blockIdx.x;
  if (first >= ntile) return;
  const int mine = static_cast<int>((ntile - first + gridDim.x - 1) / gridDim.x);
  const int total = mine * kGuChunks;
  const int64_t k0 = static_cast<int64_t>(a.s) * kGjB;
  auto tile_rc = [&](int it, int64_t &row0, int64_t &col0) {
    const int64_t tt = first + static_cast<int64_t>(it) * gridDim.x;
    const int I = static_cast<int>(tt / ncol), jx = static_cast<int>(tt % ncol);
    row0 = static_cast<int64_t>(I) * kGuM;
    col0 = static_cast<int64_t>(jx < a.s ? jx : jx + 1) * kGjB;
  };
  // chunk gc's copies: W 64 rows x 16 segments of 16 B (8 a thread), R 32 rows
  // x 64 segments (16 a thread), issued one or two at a time between the
  // tensor-core steps of the chunk before (all at once they hold up the
  // fragments' reads: the load/store unit took 12 % of the kernel's time)
  const double *lw = nullptr, *lr = nullptr;
  double *lws = nullptr, *lrs = nullptr;
  auto load_begin = [&](int gc) {
    lw = nullptr;
    if (gc >= total) return;
    int64_t row0, col0;
    tile_rc(gc / kGuChunks, row0, col0);
    const int c = gc % kGuChunks, stage = gc % kGuStages;
    lw = a.A + (row0 + (tid >> 4)) * a.ld + k0 + c * kGuKC + 2 * (tid & 15);
    lws = As + stage * kGuABuf + (tid >> 4) * kGuAS + 2 * (tid & 15);
    lr = a.R + static_cast<int64_t>(c * kGuKC + (tid >> 6)) * a.ld + col0 + 2 * (tid & 63);
    lrs = Bs + stage * kGuBBuf + (tid >> 6) * kGuBS + 2 * (tid & 63);
    // the tile's old values (none for the pivot block's rows, which become
    // Q R) on their way into L2
    if (c == 0 && (row0 < k0 || row0 >= k0 + kGjB) && tid < kGuM) {
      const double *src = a.A + (row0 + tid) * a.ld + col0;
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(static_cast<unsigned>(kGjB * sizeof(double)))
                   : "memory");
    }
  };
  auto load_w = [&](int v) {
    if (lw) cp_async16(lws + 8 * v * kGuAS, lw + 8 * v * a.ld);
  };
  auto load_r = [&](int v) {
    if (lw) cp_async16(lrs + 2 * v * kGuBS, lr + 2 * v * a.ld);
  };

  load_begin(0);
#pragma unroll
  for (int v = 0; v < 8; ++v) load_w(v);
#pragma unroll
  for (int v = 0; v < 16; ++v) load_r(v);
  cp_async_commit();
  double acc[2][8][4];
#pragma unroll
  for (int mi = 0; mi < 2; ++mi)
#pragma unroll
    for (int ni = 0; ni < 8; ++ni)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[mi][ni][i] = 0.0;
  for (int gc = 0; gc < total; ++gc) {
    cp_async_wait<0>();
    __syncthreads();
    load_begin(gc + 1);
    const int stage = gc % kGuStages;
    const bool last = gc % kGuChunks == kGuChunks - 1;
    // the tile of this chunk: old values (from L2) + W R in its epilogue, a
    // quarter (8 rows apart, 8 x 2 columns a lane) at a time, the first requested
    // before the last products and each other one before its predecessor is
    // stored
    int64_t row0, col0;
    tile_rc(gc / kGuChunks, row0, col0);
    const bool needC = row0 < k0 || row0 >= k0 + kGjB;
    double *const o = a.A + (row0 + wr + g) * a.ld + col0 + wc + 2 * t;
    double2 old[2][8];
    auto request = [&](int q) {
#pragma unroll
      for (int ni = 0; ni < 8; ++ni)
        old[q & 1][ni] = needC ? __ldcg(reinterpret_cast<const double2 *>(o + 8 * q * a.ld + 8 * ni))
                               : make_double2(0.0, 0.0);
    };
#pragma unroll
    for (int ks = 0; ks < kGuKC / 16; ++ks) {
      if (ks == 1 && last) request(0);
      const double *as = As + stage * kGuABuf + (wr + g) * kGuAS + 16 * ks + t;
      const double *bs = Bs + stage * kGuBBuf + (16 * ks + t) * kGuBS + wc + g;
      double af[2][8];
#pragma unroll
      for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int i = 0; i < 8; ++i) af[mi][i] = as[(16 * mi + 8 * (i & 1)) * kGuAS + 4 * (i >> 1)];
      // B fragments double-buffered: those of column block ni + 1 are read
      // while the tensor-core steps of column block ni issue
      double bf[2][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) bf[0][j] = bs[4 * j * kGuBS];
#pragma unroll
      for (int ni = 0; ni < 8; ++ni) {
        if (ni + 1 < 8) {
#pragma unroll
          for (int j = 0; j < 4; ++j) bf[(ni + 1) & 1][j] = bs[4 * j * kGuBS + 8 * (ni + 1)];
        }
#pragma unroll
        for (int mi = 0; mi < 2; ++mi) mma_f64_16816(acc[mi][ni], af[mi], bf[ni & 1]);
        load_r(8 * ks + ni);
        if (ks == 0) load_w(ni);
      }
    }
    cp_async_commit();  // an empty group past the end
    if (!last) continue;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (q + 1 < 4) request(q + 1);
#pragma unroll
      for (int ni = 0; ni < 8; ++ni) {
        double *c = &acc[q >> 1][ni][2 * (q & 1)];
        *reinterpret_cast<double2 *>(o + 8 * q * a.ld + 8 * ni) =
            make_double2(old[q & 1][ni].x + c[0], old[q & 1][ni].y + c[1]);
        c[0] = 0.0;
        c[1] = 0.0;
      }
    }
  }
  cp_async_wait<0>();
}

// The padding of an n x n matrix to np x np: identity (its inverse is the
// identity again, and it never mixes with the n x n part); and the
// bookkeeping arrays of the pivot-block inversions.
__global__ void gj_prepare_kernel(double *A, int64_t n, int64_t np, int64_t ld, int64_t *off, int32_t *size,
                                  int32_t *info, int steps) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t pad = np - n;
  // rows n..np-1 (all np columns), then columns n..np-1 of rows 0..n-1
  const int64_t total = pad * np + n * pad;
  for (int64_t t = t0; t < total; t += stride) {
    int64_t i, j;
    if (t < pad * np) {
      i = n + t / np;
      j = t % np;
    } else {
      i = (t - pad * np) / pad;
      j = n + (t - pad * np) % pad;
    }
    A[i * ld + j] = (i == j) ? 1.0 : 0.0;
  }
  if (t0 == 0) {
    off[0] = 0;
    size[0] = kGjB;
  }
  for (int64_t t = t0; t < steps; t += stride) info[t] = 0;
}

struct GjWorkspace {
  size_t q, r, info, off, size, bytes;
};

GjWorkspace gj_layout(int64_t np, int64_t ld) {
  GjWorkspace w{};
  size_t o = 0;
  auto take = [&](size_t nb) {
    const size_t at = o;
    o += round_up(nb, 256);
    return at;
  };
  w.q = take(static_cast<size_t>(kGjB) * kGjB * sizeof(double));
  w.r = take(static_cast<size_t>(kGjB) * static_cast<size_t>(ld) * sizeof(double));
  w.info = take(static_cast<size_t>(np / kGjB) * sizeof(int32_t));
  w.off = take(sizeof(int64_t));
  w.size = take(sizeof(int32_t));
  w.bytes = o;
  return w;
}

}  // namespace
}  // namespace f3d

extern "C" {

int f3d_dense_inverse_workspace_bytes(int64_t n, int64_t ld, size_t *bytes) {
  if (!bytes) return F3D_ERR_NULL;
  if (n < 0 || ld < 0) return F3D_ERR_SHAPE;
  const int64_t np = static_cast<int64_t>(f3d::round_up(static_cast<size_t>(n), f3d::kGjB));
  *bytes = f3d::gj_layout(np, std::max<int64_t>(ld, np)).bytes;
  return F3D_OK;
}

int f3d_dense_inverse(double *A, int64_t n, int64_t ld, void *workspace, size_t workspace_bytes, void *stream) {
  using namespace f3d;
  if (n < 0) return F3D_ERR_SHAPE;
  if (n == 0) return F3D_OK;
  if (!A || !workspace) return F3D_ERR_NULL;
  const int64_t np = static_cast<int64_t>(round_up(static_cast<size_t>(n), kGjB));
  const int64_t tiles = np / kGjB;
  if (ld < np || (ld & 1)) return F3D_ERR_SHAPE;
  if (tiles > 65535) return F3D_ERR_TOO_LARGE;
  if (!aligned(A, 16) || !aligned(workspace, 256)) return F3D_ERR_ALIGN;
  const GjWorkspace L = gj_layout(np, ld);
  if (workspace_bytes < L.bytes) return F3D_ERR_WORKSPACE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  unsigned char *w = static_cast<unsigned char *>(workspace);
  double *Q = reinterpret_cast<double *>(w + L.q), *R = reinterpret_cast<double *>(w + L.r);
  int32_t *info = reinterpret_cast<int32_t *>(w + L.info);
  int64_t *off = reinterpret_cast<int64_t *>(w + L.off);
  int32_t *size = reinterpret_cast<int32_t *>(w + L.size);

  if (cudaFuncSetAttribute(gj_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(kGjSmemPanel)) != cudaSuccess ||
      cudaFuncSetAttribute(gj_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(kGjSmemUpdate)) != cudaSuccess)
    return F3D_ERR_CUDA;
  const int64_t update_tiles = (tiles - 1) * tiles * (kGjB / kGuM);
  const unsigned update_grid = static_cast<unsigned>(std::min<int64_t>(update_tiles, 2 * static_cast<int64_t>(sm_count())));
  const int prep_blocks = static_cast<int>(std::min<int64_t>(4 * sm_count(), std::max<int64_t>(1, (np - n) * 2 * np / 256 + 1)));
  gj_prepare_kernel<<<prep_blocks, 256, 0, st>>>(A, n, np, ld, off, size, info, static_cast<int>(tiles));
  if (launch_status()) return F3D_ERR_CUDA;

  GjArgs a{};
  a.A = A;
  a.R = R;
  a.Q = Q;
  a.ld = ld;
  a.err = device_error_word();
  if (!a.err) return F3D_ERR_CUDA;
  for (int s = 0; s < tiles; ++s) {
    const int64_t k0 = static_cast<int64_t>(s) * kGjB;
    int rc = pivot_block_inverse(A + k0 * ld + k0, ld, Q, off, size, info + s, st);
    if (rc) return rc;
    a.s = s;
    gj_panel_kernel<<<static_cast<unsigned>(tiles * (kGjB / kGpM)), kGpThreads, kGjSmemPanel, st>>>(a);
    if (launch_status()) return F3D_ERR_CUDA;
    if (tiles > 1) {
      gj_update_kernel<<<update_grid, kGuThreads, kGjSmemUpdate, st>>>(a, static_cast<int>(tiles));
      if (launch_status()) return F3D_ERR_CUDA;
    }
  }
  std::vector<int32_t> h(static_cast<size_t>(tiles));
  int err = 0;
  if (cudaMemcpyAsync(h.data(), info, h.size() * sizeof(int32_t), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaMemcpyAsync(&err, a.err, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return F3D_ERR_CUDA;
  if (err != 0) {
    if (cudaMemsetAsync(a.err, 0, sizeof(int), st) != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess)
      return F3D_ERR_CUDA;
    return err;
  }
  for (int32_t v : h)
    if (v != 0) return F3D_ERR_SINGULAR;
  return F3D_OK;
}

}  // extern "C"
