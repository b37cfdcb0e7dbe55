// RBF quadrature weights of a smooth closed surface: fiber3d's
// Smooth_Closed_Surface_Quadrature_RBF with the exact surface gradient
// (python/quadratures/Smooth_Closed_Surface_Quadrature_RBF.py:3-470; the
// method of Reeger, Fornberg & Watts, Proc. R. Soc. A 472 (2016)), the
// periphery's and bodies' set-up step (tstep/tstep.py:297-300,
// body/body.py:104-107).
//
// The reference loops over triangles in Python (about 5 ms each).  Here the
// whole computation is nine kernels on one stream:
//   1. quad_prep: per triangle, sorted vertices, unit normal and midpoint;
//      its three edges go into a device hash table (key = i * n + j).
//   2. quad_edges: per triangle edge, the partner triangle from the table and
//      the edge normal, the average of the two triangles' normals (:118-127).
//   3. quad_knn: per triangle, the 80 nodes nearest its midpoint (:114-115),
//      selected exactly among the float-rounded squared distances held in
//      shared memory, ties resolved on the double distances, then index.
//      The nodes go in tiles of 24576, the best 80 carried from tile to tile.
//   4. quad_geometry: per triangle, the projection onto the triangle's plane
//      (:162-236), the exact integrals of r^7 (:262-309) and of the degree-7
//      monomials (:473-622, here by Gauss-Legendre on Green's-theorem line
//      integrals) and the area-element distortion (:431-447); quad_triangle:
//      the 116 x 116 saddle-point solve (:334-336), LU with partial pivoting in
//      shared memory, 16 columns at a time, the trailing update on the FP64
//      tensor cores, the right-hand side carried along.
//   5. quad_count / quad_scan / quad_fill / quad_sum: the per-node sum of the
//      triangle weights in triangle order (:460-468), deterministic.
#include <algorithm>
#include <climits>

#include "f3d_common.cuh"

namespace f3d {

// Node coordinates are addressed as 3 * node in 32-bit int arithmetic, so a
// surface has at most INT32_MAX / 3 nodes.
constexpr int64_t kQuadMaxNodes = 0x7fffffffLL / 3;

constexpr int kQuadNbr = 80;                 // nearest neighbours (n in the paper)
constexpr int kQuadOrder = 7;                // polynomial degree (m)
constexpr int kQuadPoly = 36;                // (m + 1)(m + 2) / 2
constexpr int kQuadDim = kQuadNbr + kQuadPoly;  // 116
constexpr int kQuadRhsCol = kQuadDim;        // column 116 holds the right-hand side
constexpr int kKnnThreads = 256;
constexpr int kKnnBins = kKnnThreads;        // of the radix select, one per thread
constexpr int kKnnCand = 256;
static_assert(kKnnBins == 256, "8 bits a pass");
constexpr int kKnnTile = 24576;             // nodes per k-NN pass (two triangles' keys in shared memory)
constexpr double kEpsMult = 1e-4;
constexpr double kDblEps = 2.220446049250313e-16;

// 6-point Gauss-Legendre on [-1, 1] (exact to degree 11).
__constant__ double kGlX[6] = {-0.9324695142031520278123016, -0.6612093864662645136613996,
                               -0.2386191860831969086305017, 0.2386191860831969086305017,
                               0.6612093864662645136613996,  0.9324695142031520278123016};
__constant__ double kGlW[6] = {0.1713244923791703450402961, 0.3607615730481386075698335,
                               0.4679139345726910473898703, 0.4679139345726910473898703,
                               0.3607615730481386075698335, 0.1713244923791703450402961};

struct QuadWs {
  int32_t *tri;     // ntri x 3, sorted vertex indices
  double *tnorm;    // ntri x 3
  double *mid;      // ntri x 3
  double *enorm;    // ntri x 9: edges (i0,i1), (i0,i2), (i1,i2)
  long long *hkey;  // hash keys (-1 empty)
  int32_t *hid;     // 2 per key: stacked edge ids (-1 empty)
  int32_t *nni;     // ntri x 80
  double *wt;       // ntri x 80: the area-element factors, then the triangles' weights
  double *rec;      // kTriRec per triangle of a chunk
  int32_t *count;   // n + 1 (exclusive offsets after the scan)
  int32_t *cursor;  // n
  int32_t *entry;   // ntri x 80
  int hbits;
};

__device__ __forceinline__ unsigned hash_slot(long long key, int hbits) {
  return static_cast<unsigned>((static_cast<unsigned long long>(key) * 0x9E3779B97F4A7C15ull) >> (64 - hbits));
}

__device__ __forceinline__ double dot3_rn(const double *a, const double *b) {
  return __dadd_rn(__dadd_rn(__dmul_rn(a[0], b[0]), __dmul_rn(a[1], b[1])), __dmul_rn(a[2], b[2]));
}

__device__ __forceinline__ void cross_rn(const double *a, const double *b, double *c) {
  c[0] = __dsub_rn(__dmul_rn(a[1], b[2]), __dmul_rn(a[2], b[1]));
  c[1] = __dsub_rn(__dmul_rn(a[2], b[0]), __dmul_rn(a[0], b[2]));
  c[2] = __dsub_rn(__dmul_rn(a[0], b[1]), __dmul_rn(a[1], b[0]));
}

// ---------------------------------------------------------------- 1. prep --
__global__ void quad_prep_kernel(const double *__restrict__ X, int n, const int32_t *__restrict__ tri_in,
                                 int ntri, QuadWs w, int *err) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntri) return;
  int i0 = tri_in[3 * t], i1 = tri_in[3 * t + 1], i2 = tri_in[3 * t + 2];
  if (i0 < 0 || i1 < 0 || i2 < 0 || i0 >= n || i1 >= n || i2 >= n) {
    record_error(err, F3D_ERR_ARG);
    i0 = 0, i1 = 0, i2 = 0;
  }
  if (i0 > i1) { const int s = i0; i0 = i1; i1 = s; }
  if (i1 > i2) { const int s = i1; i1 = i2; i2 = s; }
  if (i0 > i1) { const int s = i0; i0 = i1; i1 = s; }
  if (i0 == i1 || i1 == i2) record_error(err, F3D_ERR_ARG);
  w.tri[3 * t] = i0, w.tri[3 * t + 1] = i1, w.tri[3 * t + 2] = i2;
  double v1[3], v2[3], nrm[3];
  for (int c = 0; c < 3; ++c) {
    v1[c] = __dsub_rn(X[3 * i1 + c], X[3 * i0 + c]);
    v2[c] = __dsub_rn(X[3 * i2 + c], X[3 * i0 + c]);
  }
  // (V1 x V2) in the reference's component order (:111)
  nrm[0] = __dsub_rn(__dmul_rn(v1[1], v2[2]), __dmul_rn(v2[1], v1[2]));
  nrm[1] = __dsub_rn(__dmul_rn(v2[0], v1[2]), __dmul_rn(v1[0], v2[2]));
  nrm[2] = __dsub_rn(__dmul_rn(v1[0], v2[1]), __dmul_rn(v2[0], v1[1]));
  const double nn = __dsqrt_rn(dot3_rn(nrm, nrm));
  for (int c = 0; c < 3; ++c) {
    w.tnorm[3 * t + c] = __ddiv_rn(nrm[c], nn);
    w.mid[3 * t + c] = __ddiv_rn(__dadd_rn(__dadd_rn(X[3 * i0 + c], X[3 * i1 + c]), X[3 * i2 + c]), 3.0);
  }
  const int ea[3] = {i0, i0, i1}, eb[3] = {i1, i2, i2};
  const unsigned hmask = (1u << w.hbits) - 1u;
  for (int s = 0; s < 3; ++s) {
    const long long key = static_cast<long long>(ea[s]) * n + eb[s];
    const int id = s * ntri + t;
    unsigned slot = hash_slot(key, w.hbits);
    bool placed = false;
    for (unsigned probe = 0; probe <= hmask; ++probe) {
      const long long prev = static_cast<long long>(atomicCAS(reinterpret_cast<unsigned long long *>(w.hkey + slot),
                                                              ~0ull, static_cast<unsigned long long>(key)));
      if (prev == -1 || prev == key) {
        if (atomicCAS(w.hid + 2 * slot, -1, id) != -1 && atomicCAS(w.hid + 2 * slot + 1, -1, id) != -1)
          record_error(err, F3D_ERR_ARG);  // an edge shared by more than two triangles
        placed = true;
        break;
      }
      slot = (slot + 1) & hmask;
    }
    if (!placed) record_error(err, F3D_ERR_ARG);
  }
}

// --------------------------------------------------------------- 2. edges --
__global__ void quad_edges_kernel(int n, int ntri, QuadWs w, int *err) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= 3 * ntri) return;
  const int t = g / 3, s = g % 3;
  const int i0 = w.tri[3 * t], i1 = w.tri[3 * t + 1], i2 = w.tri[3 * t + 2];
  const int a = s == 2 ? i1 : i0, b = s == 0 ? i1 : i2;
  const long long key = static_cast<long long>(a) * n + b;
  const int id = s * ntri + t;
  const unsigned hmask = (1u << w.hbits) - 1u;
  unsigned slot = hash_slot(key, w.hbits);
  int other = -1;
  for (unsigned probe = 0; probe <= hmask; ++probe) {
    const long long k = w.hkey[slot];
    if (k == key) {
      const int p = w.hid[2 * slot], q = w.hid[2 * slot + 1];
      other = p == id ? q : (q == id ? p : -1);
      break;
    }
    if (k == -1) break;
    slot = (slot + 1) & hmask;
  }
  double e[3] = {0.0, 0.0, 0.0};
  if (other < 0) {
    record_error(err, F3D_ERR_ARG);  // an edge of only one triangle: the surface is not closed
  } else {
    // the first copy in the stacked edge order comes first in the average
    const int first = id < other ? id : other, second = id < other ? other : id;
    const double *na = w.tnorm + 3 * (first % ntri);
    const double *nb = w.tnorm + 3 * (second % ntri);
    const double d = dot3_rn(na, nb);
    const double sg = d > 0.0 ? 1.0 : (d < 0.0 ? -1.0 : 0.0);
    for (int c = 0; c < 3; ++c) e[c] = __ddiv_rn(__dadd_rn(na[c], __dmul_rn(sg, nb[c])), 2.0);
    const double en = __dsqrt_rn(dot3_rn(e, e));
    for (int c = 0; c < 3; ++c) e[c] = __ddiv_rn(e[c], en);
  }
  for (int c = 0; c < 3; ++c) w.enorm[9 * t + 3 * s + c] = e[c];
}

// ----------------------------------------------------------------- 3. kNN --
__device__ __forceinline__ unsigned fkey(double d) { return __float_as_uint(__double2float_rn(d)); }

// Squared distance of node g from q, rounded operation by operation.
__device__ __forceinline__ double dist2_rn(const double *__restrict__ X, int g, const double (&q)[3]) {
  const double dx = __dsub_rn(q[0], X[3 * g]), dy = __dsub_rn(q[1], X[3 * g + 1]), dz = __dsub_rn(q[2], X[3 * g + 2]);
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

// The 80th smallest of m float keys by a radix select (8 bits a pass), the
// whole CTA.
__device__ unsigned knn_radix_select(const unsigned *keys, int m, int *hist, int *s_part, int *s_bin, int *s_below) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned prefix = 0;
  int kk = kQuadNbr;  // rank (1-based) still to find among keys matching the prefix
  for (int shift = 24; shift >= 0; shift -= 8) {
    hist[tid] = 0;
    __syncthreads();
    for (int pb = 0; pb < m; pb += kKnnThreads) {
      const int j = pb + tid;
      int bin = -1 - lane;  // distinct per lane when not counted
      if (j < m) {
        const unsigned key = keys[j];
        if (shift == 24 || (key >> (shift + 8)) == prefix) bin = static_cast<int>((key >> shift) & 255u);
      }
      const unsigned peers = __match_any_sync(0xffffffffu, bin);
      if (bin >= 0 && lane == __ffs(peers) - 1) atomicAdd(hist + bin, __popc(peers));
    }
    __syncthreads();
    // the bin where the running count reaches kk
    const int local = hist[tid];
    int incl = local;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) s_part[warp] = incl;
    __syncthreads();
    int before = 0;
    for (int w2 = 0; w2 < warp; ++w2) before += s_part[w2];
    const int excl = before + incl - local;
    if (excl < kk && excl + local >= kk) {
      *s_bin = tid;
      *s_below = excl;
    }
    __syncthreads();
    prefix = (prefix << 8) | static_cast<unsigned>(*s_bin);
    kk -= *s_below;
    __syncthreads();
  }
  return prefix;
}

// Two triangles per CTA, so that each node is loaded once for both; the first
// 128 threads select for the first, the others for the second.  The nodes are
// taken in tiles of `tile`: each tile's squared distances, rounded to float
// (a monotone key), go to shared memory together with the best 80 of the
// earlier tiles, so a surface of any size fits; a surface of at most `tile`
// nodes is one pass.
//
// What bounds it is the passes over the keys.  The threshold comes without a
// histogram: the 80th smallest of the minima of 128 disjoint groups of keys
// (two threads' each) is no smaller than the 80th smallest key, and for nodes
// spread over the groups only about 128 ln(128/48) = 125 keys lie at or below
// it.  One more pass collects those; their exact (distance, index) ranks are
// found by counting.  Where more than kKnnCand nodes pass (many nodes of one
// group close by, or equal distances), the radix select finds the exact
// threshold.  24500 triangles x 12252 nodes: 1.09 ms, against 5.35 ms for the
// radix select on every triangle and a bitonic sort of the candidates; 2880 x
// 1442: 71 against 105 us.
__global__ void __launch_bounds__(kKnnThreads) quad_knn_kernel(const double *__restrict__ X, int n,
                                                               const double *__restrict__ mid, int ntri, int tile,
                                                               int32_t *__restrict__ nni, int *err) {
  extern __shared__ __align__(16) unsigned char knn_smem[];
  constexpr int kHalf = kKnnThreads / 2;
  double(*pd)[kQuadNbr] = reinterpret_cast<double(*)[kQuadNbr]>(knn_smem);        // [2]: the earlier tiles' best
  double(*cd)[kKnnCand] = reinterpret_cast<double(*)[kKnnCand]>(pd + 2);          // [2]: candidate distances
  int(*cj)[kKnnCand] = reinterpret_cast<int(*)[kKnnCand]>(cd + 2);                // [2]: and indices
  int(*pj)[kQuadNbr] = reinterpret_cast<int(*)[kQuadNbr]>(cj + 2);                // [2]
  int *hist = reinterpret_cast<int *>(pj + 2);                                    // kKnnBins
  unsigned *keys0 = reinterpret_cast<unsigned *>(hist + kKnnBins);                // [2][tile + 80]
  __shared__ __align__(16) unsigned s_min[2][kHalf];  // read four at a time
  __shared__ unsigned s_tau[2];
  __shared__ int s_part[kKnnThreads / 32];
  __shared__ int s_bin, s_below, s_ncand[2];
  const int tid = threadIdx.x;
  const int h = tid / kHalf, u = tid % kHalf;  // this thread's triangle in the selection, its place there
  const int stride = (tile + kQuadNbr + 3) & ~3;
  for (int t0 = 2 * blockIdx.x; t0 < ntri; t0 += 2 * gridDim.x) {
    const int t1 = min(t0 + 1, ntri - 1);
    const double qa[3] = {mid[3 * t0], mid[3 * t0 + 1], mid[3 * t0 + 2]};
    const double qb[3] = {mid[3 * t1], mid[3 * t1 + 1], mid[3 * t1 + 2]};
    int nprev = 0;
    for (int base = 0; base < n; base += tile) {
      const int tl = min(tile, n - base);
      unsigned ma = 0xffffffffu, mb = 0xffffffffu;
#pragma unroll 4
      for (int j = tid; j < tl; j += kKnnThreads) {
        const unsigned ka = fkey(dist2_rn(X, base + j, qa)), kb = fkey(dist2_rn(X, base + j, qb));
        keys0[j] = ka;
        keys0[stride + j] = kb;
        ma = min(ma, ka);
        mb = min(mb, kb);
      }
      if (tid < nprev) {
        const unsigned ka = fkey(pd[0][tid]), kb = fkey(pd[1][tid]);
        keys0[tl + tid] = ka;
        keys0[stride + tl + tid] = kb;
        ma = min(ma, ka);
        mb = min(mb, kb);
      }
      const int m = tl + nprev;  // >= 80: the first tile has min(n, tile) >= 80 nodes
      ma = min(ma, __shfl_xor_sync(0xffffffffu, ma, 1));
      mb = min(mb, __shfl_xor_sync(0xffffffffu, mb, 1));
      if ((tid & 1) == 0) {
        s_min[0][tid >> 1] = ma;
        s_min[1][tid >> 1] = mb;
      }
      if (tid < 2) s_ncand[tid] = 0;
      __syncthreads();
      {
        const unsigned mine = s_min[h][u];
        int below = 0;
        for (int q = 0; q < kHalf; q += 4) {
          const uint4 o = *reinterpret_cast<const uint4 *>(&s_min[h][q]);
          below += (o.x < mine || (o.x == mine && q < u)) + (o.y < mine || (o.y == mine && q + 1 < u)) +
                   (o.z < mine || (o.z == mine && q + 2 < u)) + (o.w < mine || (o.w == mine && q + 3 < u));
        }
        if (below == kQuadNbr - 1) s_tau[h] = mine;
      }
      __syncthreads();
      // every key at or below the threshold is a candidate (its place first;
      // distances and indices follow for all candidates at once)
      auto collect = [&](int q, unsigned tau, int from, int step) {
        const uint4 *keys = reinterpret_cast<const uint4 *>(keys0 + q * stride);
        auto take = [&](unsigned key, int j) {
          if (key <= tau && j < m) {
            const int slot = atomicAdd(&s_ncand[q], 1);
            if (slot < kKnnCand) cj[q][slot] = j;
          }
        };
#pragma unroll 2
        for (int j = from; j < (m + 3) / 4; j += step) {
          const uint4 k = keys[j];
          if (min(min(k.x, k.y), min(k.z, k.w)) <= tau) {
            take(k.x, 4 * j);
            take(k.y, 4 * j + 1);
            take(k.z, 4 * j + 2);
            take(k.w, 4 * j + 3);
          }
        }
      };
      collect(h, s_tau[h], u, kHalf);
      __syncthreads();
      for (int q = 0; q < 2; ++q) {
        if (s_ncand[q] <= kKnnCand) continue;
        const unsigned tau = knn_radix_select(keys0 + q * stride, m, hist, s_part, &s_bin, &s_below);
        if (tid == 0) s_ncand[q] = 0;
        __syncthreads();
        collect(q, tau, tid, kKnnThreads);
        __syncthreads();
        if (s_ncand[q] > kKnnCand && tid == 0) record_error(err, F3D_ERR_TOO_LARGE);
      }
      for (int q = 0; q < 2; ++q) {
        if (tid < min(s_ncand[q], kKnnCand)) {
          const int j = cj[q][tid];
          cd[q][tid] = j < tl ? dist2_rn(X, base + j, q ? qb : qa) : pd[q][j - tl];
          cj[q][tid] = j < tl ? base + j : pj[q][j - tl];
        }
      }
      __syncthreads();
      // the candidates' places by (distance, index); the 80 best are the
      // result, or go on to the next tile
      const int nc = min(s_ncand[h], kKnnCand);
      const bool last = base + tile >= n;
      for (int c = u; c < nc; c += kHalf) {
        const double d = cd[h][c];
        const unsigned long long mine = static_cast<unsigned long long>(__double_as_longlong(d));
        const int j = cj[h][c];
        int at = 0;
#pragma unroll 8
        for (int o = 0; o < nc; ++o) {  // no branch: the lanes' outcomes differ
          const unsigned long long ob = static_cast<unsigned long long>(__double_as_longlong(cd[h][o]));
          at += static_cast<int>(ob < mine) | (static_cast<int>(ob == mine) & static_cast<int>(cj[h][o] < j));
        }
        if (at < kQuadNbr) {
          if (last) {
            if (t0 + h < ntri) nni[static_cast<int64_t>(t0 + h) * kQuadNbr + at] = j < n ? j : 0;
          } else {
            pd[h][at] = d;
            pj[h][at] = j;
          }
        }
      }
      nprev = kQuadNbr;
      __syncthreads();
    }
  }
}

// ------------------------------------------------------------ 4. triangle --
// Integral of r^7 over the right triangle with legs alpha and beta (:302).
__device__ __forceinline__ double rbf_right_triangle(double a, double b) {
  const double a2 = a * a, b2 = b * b;
  return a * (b * sqrt(a2 + b2) * (279.0 * a2 * a2 * a2 + 326.0 * a2 * a2 * b2 + 200.0 * a2 * b2 * b2 + 48.0 * b2 * b2 * b2) +
              105.0 * (a2 * a2) * (a2 * a2) * asinh(b / a)) /
         3456.0;
}

__device__ __forceinline__ double sgn(double x) { return x > 0.0 ? 1.0 : (x < 0.0 ? -1.0 : 0.0); }

// The projection and the right-hand side of each triangle t of [t_lo, t_hi):
// the projected centres (80 x 2) and the integrals (116) to its record, the
// area-element factors to its 80 entries of w.wt.  Mostly serial chains of
// divisions, square roots and asinh over at most 116 threads, so it is a
// kernel of its own with many CTAs per SM (0.43 ms at 24500 triangles); inside
// the elimination kernel the chains ran with nothing beside them.
constexpr int kGeoThreads = 128;
constexpr int kTriRec = 2 * kQuadNbr + kQuadDim;

struct GeoShared {
  double c[kQuadNbr][2];  // projected, shifted centres
  double l[kQuadNbr], ys[kQuadNbr];
  double xp[3], rot[9], shift[2], v[3][2], height;
};

__global__ void __launch_bounds__(kGeoThreads) quad_geometry_kernel(const double *__restrict__ X,
                                                                    const double *__restrict__ grad, int t_lo,
                                                                    QuadWs w) {
  __shared__ GeoShared S;
  const int tid = threadIdx.x;
  const int t = t_lo + static_cast<int>(blockIdx.x);
  double *rec = w.rec + static_cast<int64_t>(blockIdx.x) * kTriRec;
  const int *tv = w.tri + 3 * t;
  const double *nrm = w.tnorm + 3 * t;
  const int32_t *nb = w.nni + static_cast<int64_t>(t) * kQuadNbr;
  if (tid == 0) {
    // projection point (:162-201)
    double A[3], B[3], C[3], AB[3], BC[3], CA[3];
    for (int c = 0; c < 3; ++c) {
      A[c] = X[3 * tv[0] + c], B[c] = X[3 * tv[1] + c], C[c] = X[3 * tv[2] + c];
      AB[c] = __dsub_rn(B[c], A[c]), BC[c] = __dsub_rn(C[c], B[c]), CA[c] = __dsub_rn(A[c], C[c]);
    }
    const double *nAB = w.enorm + 9 * t, *nCA = nAB + 3, *nBC = nAB + 6;
    double nOAB[3], nOBC[3], nOCA[3], vOA[3];
    cross_rn(nAB, AB, nOAB);
    cross_rn(nBC, BC, nOBC);
    cross_rn(nCA, CA, nOCA);
    cross_rn(nOAB, nOCA, vOA);
    const double tA = __ddiv_rn(dot3_rn(nOBC, AB), dot3_rn(nOBC, vOA));
    for (int c = 0; c < 3; ++c) S.xp[c] = __dadd_rn(A[c], __dmul_rn(tA, vOA[c]));
    // rotation taking the normal to +z (:210-220)
    const double rxy = __dsqrt_rn(__dadd_rn(__dmul_rn(nrm[0], nrm[0]), __dmul_rn(nrm[1], nrm[1])));
    if (rxy < kDblEps) {
      for (int i = 0; i < 9; ++i) S.rot[i] = (i % 4 == 0) ? 1.0 : 0.0;
    } else {
      const double nn = __dsqrt_rn(dot3_rn(nrm, nrm));
      const double r1[9] = {__ddiv_rn(nrm[2], nn), 0.0, -__ddiv_rn(rxy, nn), 0.0, 1.0, 0.0,
                            __ddiv_rn(rxy, nn), 0.0, __ddiv_rn(nrm[2], nn)};
      const double r2[9] = {__ddiv_rn(nrm[0], rxy), __ddiv_rn(nrm[1], rxy), 0.0, -__ddiv_rn(nrm[1], rxy),
                            __ddiv_rn(nrm[0], rxy), 0.0, 0.0, 0.0, 1.0};
      for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j)
          S.rot[3 * i + j] = __dadd_rn(__dadd_rn(__dmul_rn(r1[3 * i], r2[j]), __dmul_rn(r1[3 * i + 1], r2[3 + j])),
                                       __dmul_rn(r1[3 * i + 2], r2[6 + j]));
    }
    double d[3];
    for (int c = 0; c < 3; ++c) d[c] = __dsub_rn(w.mid[3 * t + c], S.xp[c]);
    S.shift[0] = dot3_rn(S.rot, d);
    S.shift[1] = dot3_rn(S.rot + 3, d);
    const double *V[3] = {A, B, C};
    for (int r = 0; r < 3; ++r) {
      for (int c = 0; c < 3; ++c) d[c] = __dsub_rn(V[r][c], S.xp[c]);
      S.v[r][0] = __dsub_rn(dot3_rn(S.rot, d), S.shift[0]);
      S.v[r][1] = __dsub_rn(dot3_rn(S.rot + 3, d), S.shift[1]);
    }
  }
  __syncthreads();
  if (tid < kQuadNbr) {
    // project neighbour tid into the plane (:225-236)
    const int j = nb[tid];
    double Q[3], d[3], p[3];
    for (int c = 0; c < 3; ++c) Q[c] = X[3 * j + c];
    const double A0 = X[3 * tv[0]], A1 = X[3 * tv[0] + 1], A2 = X[3 * tv[0] + 2];
    const double num = __dadd_rn(__dadd_rn(__dmul_rn(nrm[0], __dsub_rn(A0, Q[0])), __dmul_rn(nrm[1], __dsub_rn(A1, Q[1]))),
                                 __dmul_rn(nrm[2], __dsub_rn(A2, Q[2])));
    for (int c = 0; c < 3; ++c) d[c] = __dsub_rn(Q[c], S.xp[c]);
    const double mult = __ddiv_rn(num, dot3_rn(nrm, d));
    for (int c = 0; c < 3; ++c) p[c] = __dsub_rn(__dadd_rn(Q[c], __dmul_rn(mult, d[c])), S.xp[c]);
    const double u0 = dot3_rn(S.rot, p), u1 = dot3_rn(S.rot + 3, p), u2 = dot3_rn(S.rot + 6, p);
    if (tid == 0) S.height = u2;
    const double cx = __dsub_rn(u0, S.shift[0]), cy = __dsub_rn(u1, S.shift[1]);
    S.c[tid][0] = cx, S.c[tid][1] = cy;
    rec[2 * tid] = cx, rec[2 * tid + 1] = cy;
    // area-element distortion (:431-442)
    const double *g = grad + 3 * j;
    const double gn = __dsqrt_rn(dot3_rn(g, g));
    const double nv = __dsqrt_rn(dot3_rn(d, d));
    double vh[3], ns[3];
    for (int c = 0; c < 3; ++c) vh[c] = __ddiv_rn(d[c], nv), ns[c] = __ddiv_rn(g[c], gn);
    const double pn = __dsqrt_rn(dot3_rn(nrm, nrm));
    double pu[3];
    for (int c = 0; c < 3; ++c) pu[c] = __ddiv_rn(nrm[c], pn);
    S.ys[tid] = __ddiv_rn(dot3_rn(pu, vh), dot3_rn(ns, vh));  // ratio of the normal projections
    S.l[tid] = nv;
  }
  __syncthreads();
  if (tid < kQuadNbr) {
    const double cx = __dadd_rn(S.c[tid][0], S.shift[0]), cy = __dadd_rn(S.c[tid][1], S.shift[1]);
    const double R = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(cx, cx), __dmul_rn(cy, cy)), __dmul_rn(S.height, S.height)));
    const double rr = __ddiv_rn(S.l[tid], R);
    w.wt[static_cast<int64_t>(t) * kQuadNbr + tid] = fabs(__dmul_rn(S.ys[tid], __dmul_rn(rr, rr)));
    // exact integral of r^7 centred at this node over the triangle (:262-309)
    const double c0 = S.c[tid][0], c1 = S.c[tid][1];
    const double(*V)[2] = S.v;
    const double sabc = sgn(__dadd_rn(__dmul_rn(__dsub_rn(V[0][1], V[1][1]), __dsub_rn(V[2][0], V[0][0])),
                                      __dmul_rn(__dsub_rn(V[1][0], V[0][0]), __dsub_rn(V[2][1], V[0][1]))));
    double irbf = 0.0;
    for (int s = 0; s < 3; ++s) {
      const double *p1 = V[s], *p2 = V[(s + 1) % 3];
      const double ex = __dsub_rn(p2[0], p1[0]), ey = __dsub_rn(p2[1], p1[1]);
      const double m = __ddiv_rn(__dadd_rn(__dmul_rn(__dsub_rn(c0, p1[0]), ex), __dmul_rn(__dsub_rn(c1, p1[1]), ey)),
                                 __dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey)));
      const double fx = __dadd_rn(__dmul_rn(m, ex), p1[0]), fy = __dadd_rn(__dmul_rn(m, ey), p1[1]);
      const double sg1 = sabc * sgn(__dadd_rn(__dmul_rn(__dsub_rn(c1, p1[1]), __dsub_rn(fx, c0)),
                                              __dmul_rn(__dsub_rn(p1[0], c0), __dsub_rn(fy, c1))));
      const double sg2 = sabc * sgn(__dadd_rn(__dmul_rn(__dsub_rn(c1, fy), __dsub_rn(p2[0], c0)),
                                              __dmul_rn(__dsub_rn(fx, c0), __dsub_rn(p2[1], c1))));
      const double ax = __dsub_rn(c0, fx), ay = __dsub_rn(c1, fy);
      const double alpha = __dsqrt_rn(__dadd_rn(__dmul_rn(ax, ax), __dmul_rn(ay, ay)));
      const double b1x = __dsub_rn(fx, p1[0]), b1y = __dsub_rn(fy, p1[1]);
      const double b2x = __dsub_rn(fx, p2[0]), b2y = __dsub_rn(fy, p2[1]);
      const double beta1 = __dsqrt_rn(__dadd_rn(__dmul_rn(b1x, b1x), __dmul_rn(b1y, b1y)));
      const double beta2 = __dsqrt_rn(__dadd_rn(__dmul_rn(b2x, b2x), __dmul_rn(b2y, b2y)));
      const double tiny = kEpsMult * kDblEps;
      if (alpha > tiny && beta1 > tiny) irbf += sg1 * rbf_right_triangle(alpha, beta1);
      if (alpha > tiny && beta2 > tiny) irbf += sg2 * rbf_right_triangle(alpha, beta2);
    }
    rec[2 * kQuadNbr + tid] = irbf;
  } else if (tid < kQuadDim) {
    // polynomial moment m = tid - 80 of the triangle (Green's theorem,
    // Gauss-Legendre along each side)
    const int m = tid - kQuadNbr;
    int dg = 0;
    while ((dg + 1) * (dg + 2) / 2 <= m) ++dg;
    const int k = m - dg * (dg + 1) / 2, a = dg - k;
    const double(*V)[2] = S.v;
    const double sabc = sgn(__dadd_rn(__dmul_rn(__dsub_rn(V[0][1], V[1][1]), __dsub_rn(V[2][0], V[0][0])),
                                      __dmul_rn(__dsub_rn(V[1][0], V[0][0]), __dsub_rn(V[2][1], V[0][1]))));
    double acc = 0.0;
    for (int s = 0; s < 3; ++s) {
      const double *p1 = V[s], *p2 = V[(s + 1) % 3];
      const double ex = p2[0] - p1[0], ey = p2[1] - p1[1];
      double line = 0.0;
      for (int q = 0; q < 6; ++q) {
        const double tq = 0.5 * (kGlX[q] + 1.0);
        const double xq = p1[0] + tq * ex, yq = p1[1] + tq * ey;
        double v = 0.5 * kGlW[q];
        for (int e = 0; e <= a; ++e) v *= xq;
        for (int e = 0; e < k; ++e) v *= yq;
        line += v;
      }
      acc += ey * line / (a + 1);
    }
    rec[2 * kQuadNbr + tid] = sabc * acc;
  }
}

// The 116 x 116 saddle-point system of each triangle: LU with partial pivoting
// (LAPACK's choice of pivots), the right-hand side carried along as column
// 116, and back substitution.
//
// The chain of 116 pivots bounds it (the 0.5 Mflop of a triangle are 8000
// tensor-core cycles), so two triangles share an SM: a CTA is 256 threads, at
// most 128 registers and the matrix in 110 KB of shared memory, with
// everything else in the 5.5 KB that two such CTAs leave.  That is why
//  * panels are 16 columns whose rows (one per thread) go through the 16
//    pivots in registers, with one barrier per pivot;
//  * U12 and L21 stay where they are in the matrix, and the trailing update
//    (16 x 16 outputs per warp at a time, on the FP64 tensor cores) reads its
//    operands there;
//  * rows are never exchanged: `phys` maps positions to rows, a pivot is the
//    first position of largest magnitude, and the trailing rows are gathered
//    by position;
//  * half of the warps work on a panel; the others meanwhile apply the panel
//    before to the columns after it (all first apply it to this panel's).
// Row stride 118 doubles: a thread's 16-byte reads of its own row are free of
// bank conflicts, the tensor-core fragments' two-way at worst.
// The panels' transformations are not applied as explicit products (blocked
// Gauss-Jordan, which needs no back substitution): these systems have
// condition numbers near 1e17, and on a 200-node sphere of radius 0.5 that
// moved the weights by 7e-8.
// 24500 triangles: 6.9 ms (7.2 with 64-bit keys posted in three words; 7.7
// also without the look-ahead and with quotients on the chain of back
// substitution), against 27.9 ms for unblocked Gauss-Jordan with the matrix in
// the registers of one CTA per SM, two barriers per pivot.
constexpr int kTriThreads = 256;
constexpr int kTriWarps = kTriThreads / 32;
constexpr int kTriS = kQuadDim + 2;  // row stride: 116 columns, the right-hand side, one of padding
constexpr int kTriPW = 4;            // warps with panel rows
constexpr size_t kTriSmem = static_cast<size_t>(kQuadDim) * kTriS * sizeof(double);

struct TriShared {
  __align__(16) double cand[2][kTriPW][16];  // each warp's best row, by step parity
  __align__(16) double l11[16][16];          // column-major unit lower triangle of the panel
  uint4 post[2][kTriPW];                     // its candidate's trailing word, position, and reciprocal
  double c[kQuadNbr][2];                     // projected centres; then the unknowns
  __align__(16) unsigned hi[2][kTriPW];      // the candidate's key
  int phys[2][kQuadDim];                     // row at each position still to be reduced, by panel parity
  int fin[kQuadDim];                         // row of each pivot
};

// sqrt(x^7) = x^3 sqrt(x) (x >= 0; NaN below): the cube as a two-term sum, so
// that the result has the square root's rounding and its own.
__device__ __forceinline__ double sqrt_pow7(double x) {
  const double t = x * x, te = fma(x, x, -t);
  const double c = t * x, ce = fma(te, x, fma(t, x, -c));
  const double s = sqrt(x), p = c * s;
  return p + fma(ce, s, fma(c, s, -p));
}

// Pivot k = c0 + jj of the panel (jj static) on the rows in v.
template <int jj>
__device__ __forceinline__ void tri_pivot(double (&v)[16], TriShared &S, int k, bool &done, int &pos, int lane,
                                          int warp, int *err) {
  constexpr int par = jj & 1;
  // this row's candidacy: 0 none, 1 a NaN, else the leading word of |a| plus 2
  const unsigned mag = static_cast<unsigned>(__double2hiint(v[jj])) & 0x7fffffffu;
  const bool nan = v[jj] != v[jj];
  const unsigned hi = done ? 0u : (nan ? 1u : mag + 2u), lo = nan ? 0u : __double2loint(v[jj]);
  // beside the search; of zero or not a number, the error below, as of 1
  const double rcp = fabs(v[jj]) > 0.0 ? 1.0 / v[jj] : 1.0;
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
    for (int j = jj & ~1; j < 16; j += 2)
      *reinterpret_cast<double2 *>(&S.cand[par][warp][j]) = make_double2(v[j], v[j + 1]);
  }
  asm volatile("bar.sync 1, %0;" ::"n"(32 * kTriPW) : "memory");
  // the best warp
  const uint4 h = *reinterpret_cast<const uint4 *>(S.hi[par]);
  const unsigned top = max(max(h.x, h.y), max(h.z, h.w));
  int bw = h.x == top ? 0 : (h.y == top ? 1 : (h.z == top ? 2 : 3));
  if ((h.x == top) + (h.y == top) + (h.z == top) + (h.w == top) > 1) {
    // equal leading words: the rest of the key, then the position
    for (int w = bw + 1; w < kTriPW; ++w) {
      if (S.hi[par][w] != top) continue;
      const uint4 pw = S.post[par][w], pb = S.post[par][bw];
      if (pw.x > pb.x || (pw.x == pb.x && static_cast<int>(pw.y) < static_cast<int>(pb.y))) bw = w;
    }
  }
  const uint4 post = S.post[par][bw];
  const int pp = static_cast<int>(post.y);
  const double *prow = S.cand[par][bw];
  const double d = prow[jj], rd = __hiloint2double(static_cast<int>(post.w), static_cast<int>(post.z));
  if (pos == pp) {  // the pivot row
    pos = k;
    done = true;
    if (!(fabs(d) > 0.0)) {  // zero or not a number: an error; go on as if the pivot were 1 (rd is)
      record_error(err, F3D_ERR_SINGULAR);
      v[jj] = 1.0;
    }
  } else if (pos == k) {
    pos = pp;
  }
  if (!done) {
    const double l = v[jj] * rd;
    v[jj] = l;
#pragma unroll
    for (int j = jj + 1; j < 16; ++j) v[j] = fma(-l, prow[j], v[j]);
  }
}

template <int jj>
__device__ __forceinline__ void tri_panel(double (&v)[16], TriShared &S, int c0, int nb, bool &done, int &pos,
                                          int lane, int warp, int *err) {
  if constexpr (jj < 16) {
    if (jj >= nb) return;
    tri_pivot<jj>(v, S, c0 + jj, done, pos, lane, warp, err);
    tri_panel<jj + 1>(v, S, c0, nb, done, pos, lane, warp, err);
  }
}

__global__ void __launch_bounds__(kTriThreads, 2) quad_triangle_kernel(int t_lo, int count, QuadWs w, int *err) {
  extern __shared__ __align__(16) double tri_smem[];
  __shared__ TriShared S;
  double *X = tri_smem;  // [116][kTriS]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int it = blockIdx.x; it < count; it += gridDim.x) {
    const double *rec = w.rec + static_cast<int64_t>(it) * kTriRec;
    for (int i = tid; i < 2 * kQuadNbr; i += kTriThreads) (&S.c[0][0])[i] = rec[i];
    if (tid < kQuadDim) {
      *reinterpret_cast<double2 *>(X + tid * kTriS + kQuadRhsCol) = make_double2(rec[2 * kQuadNbr + tid], 0.0);
      S.phys[0][tid] = tid;
    }
    __syncthreads();
    // [Phi P; P^T 0]
    if (tid < kQuadNbr) {  // monomials by the reference's recursion (:324-329)
      const double cx = S.c[tid][0], cy = S.c[tid][1];
      double below[kQuadOrder + 1], row[kQuadOrder + 1];
      row[0] = 1.0;
#pragma unroll
      for (int dg = 0; dg <= kQuadOrder; ++dg) {
        if (dg > 0) {
#pragma unroll
          for (int k = 0; k <= dg; ++k)
            row[k] = (k >= (dg + 1) / 2) ? __dmul_rn(cy, below[k - 1]) : __dmul_rn(cx, below[k]);
        }
#pragma unroll
        for (int k = 0; k <= dg; ++k) {
          const int m = kQuadNbr + dg * (dg + 1) / 2 + k;
          X[tid * kTriS + m] = row[k];
          X[m * kTriS + tid] = row[k];
          below[k] = row[k];
        }
      }
    } else {
      for (int e = tid - kQuadNbr; e < kQuadPoly * kQuadPoly; e += kTriThreads - kQuadNbr)
        X[(kQuadNbr + e / kQuadPoly) * kTriS + kQuadNbr + e % kQuadPoly] = 0.0;
    }
    for (int e = tid; e < kQuadNbr * kQuadNbr; e += kTriThreads) {
      const int i = e / kQuadNbr, j = e % kQuadNbr;
      const double xi = S.c[i][0], yi = S.c[i][1], xj = S.c[j][0], yj = S.c[j][1];
      const double di = __dadd_rn(__dmul_rn(xi, xi), __dmul_rn(yi, yi));
      const double dj = __dadd_rn(__dmul_rn(xj, xj), __dmul_rn(yj, yj));
      const double ip = __dadd_rn(__dmul_rn(xi, xj), __dmul_rn(yi, yj));
      X[i * kTriS + j] = sqrt_pow7(__dsub_rn(__dadd_rn(dj, di), __dmul_rn(2.0, ip)));
    }
    __syncthreads();

    // The update by panel c0 of the columns [c, ce), c a multiple of 16 past
    // cs: items of 16 x 16 outputs to warps w0, w0 + 1, ...
    auto update = [&](int c0, const int *phys, int c_lo, int ce, int w0) {
      const int g = lane >> 2, t = lane & 3;
      const int cs = c0 + 16, m2 = kQuadDim - cs, rts = (m2 + 15) / 16, cts = (ce - c_lo + 15) / 16;
      for (int it2 = warp - w0; it2 < rts * cts; it2 += kTriWarps - w0) {
        const int rt = it2 % rts, c = c_lo + 16 * (it2 / rts);
        const int p0 = 16 * rt + g, p1 = p0 + 8;
        double *x0 = X + phys[cs + min(p0, m2 - 1)] * kTriS, *x1 = X + phys[cs + min(p1, m2 - 1)] * kTriS;
        double af[8], bf[2][4];
#pragma unroll
        for (int q = 0; q < 8; ++q) af[q] = -((q & 1) ? x1 : x0)[c0 + t + 4 * (q >> 1)];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double *u = X + S.fin[c0 + t + 4 * j] * kTriS;
#pragma unroll
          for (int ni = 0; ni < 2; ++ni) bf[ni][j] = u[min(c + 8 * ni + g, kQuadRhsCol)];
        }
#pragma unroll
        for (int ni = 0; ni < 2; ++ni) {
          const int cc = c + 8 * ni + 2 * t;  // this lane's two columns (the second may be the padding)
          const bool cv = cc < ce;
          double2 o0 = make_double2(0.0, 0.0), o1 = o0;
          if (cv) {
            o0 = *reinterpret_cast<const double2 *>(x0 + cc);
            o1 = *reinterpret_cast<const double2 *>(x1 + cc);
          }
          double dd[4] = {o0.x, o0.y, o1.x, o1.y};
          mma_f64_16816(dd, af, bf[ni]);
          if (cv) {
            if (p0 < m2) *reinterpret_cast<double2 *>(x0 + cc) = make_double2(dd[0], dd[1]);
            if (p1 < m2) *reinterpret_cast<double2 *>(x1 + cc) = make_double2(dd[2], dd[3]);
          }
        }
      }
    };
    for (int c0 = 0, par = 0; c0 < kQuadDim; c0 += 16, par ^= 1) {
      const int nb = min(16, kQuadDim - c0), m = kQuadDim - c0;
      // warps 0-3: the panel, from the row order of parity par to the other;
      // warps 4-7 meanwhile: the previous panel's update of the columns after
      // this one
      if (warp < kTriPW) {
        const bool live = tid < m;
        bool done = !live;
        int pos = live ? c0 + tid : INT_MAX;
        const int row = live ? S.phys[par][pos] : 0;
        double v[16];
        double *x = X + row * kTriS + c0;
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          double2 a = make_double2(0.0, 0.0);
          if (j < nb) a = *reinterpret_cast<const double2 *>(x + j);
          v[j] = a.x;
          v[j + 1] = a.y;
        }
        tri_panel<0>(v, S, c0, nb, done, pos, lane, warp, err);
        if (live) {
#pragma unroll
          for (int j = 0; j < 16; j += 2)
            if (j < nb) *reinterpret_cast<double2 *>(x + j) = make_double2(v[j], v[j + 1]);
          if (pos < c0 + nb) {
            S.fin[pos] = row;
#pragma unroll
            for (int j = 0; j < 16; ++j) S.l11[j][pos - c0] = v[j];
          } else {
            S.phys[par ^ 1][pos] = row;
          }
        }
      } else if (c0 > 0) {
        update(c0 - 16, S.phys[par], c0 + 16, kQuadRhsCol + 1, kTriPW);
      }
      __syncthreads();
      // U12 = L11^-1 A12, a column per thread (the right-hand side the last)
      const int cs = c0 + nb;
      if (tid <= kQuadRhsCol - cs) {
        double u[16];
        double *xc = X + cs + tid;
#pragma unroll
        for (int i = 0; i < 16; ++i) u[i] = i < nb ? xc[S.fin[min(c0 + i, kQuadDim - 1)] * kTriS] : 0.0;
#pragma unroll
        for (int i = 0; i < 15; ++i) {
          if (i >= nb) break;
#pragma unroll
          for (int r = i + 1; r < 16; ++r)
            if (r < nb) u[r] = fma(-S.l11[i][r], u[i], u[r]);
        }
#pragma unroll
        for (int i = 1; i < 16; ++i)
          if (i < nb) xc[S.fin[min(c0 + i, kQuadDim - 1)] * kTriS] = u[i];
      }
      __syncthreads();
      // A22 -= L21 U12 on the next panel's columns, all warps (the last
      // panel's columns are 112-115 and come with the right-hand side)
      if (cs < kQuadDim) {
        update(c0, S.phys[par ^ 1], cs, cs + 16 < kQuadDim ? cs + 16 : kQuadRhsCol + 1, 0);
        __syncthreads();
      }
    }
    // back substitution by blocks of 16: the warp that holds the block's
    // positions solves its triangle, then every earlier position takes the
    // block's unknowns out (x stays in S.c)
    if (warp < kTriPW) {
      double *xs = &S.c[0][0];
      const int k = tid;
      const double *u = X + S.fin[min(k, kQuadDim - 1)] * kTriS;
      // the row over its diagonal entry, so that the chain of unknowns is one
      // product and one exchange each
      const double rd = k < kQuadDim ? 1.0 / u[k] : 1.0;
      double y = k < kQuadDim ? u[kQuadRhsCol] * rd : 0.0;
      for (int c0 = (kQuadDim - 1) / 16 * 16; c0 >= 0; c0 -= 16) {
        const int nb = min(16, kQuadDim - c0);
        if (warp == c0 / 32) {
          double us[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) us[j] = (j < nb && k >= c0 && k < c0 + j) ? -u[c0 + j] * rd : 0.0;
#pragma unroll
          for (int j = 15; j >= 0; --j)
            if (j < nb) y = fma(us[j], __shfl_sync(0xffffffffu, y, (c0 + j) & 31), y);
          if (k >= c0 && k < c0 + nb) xs[k] = y;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kTriPW) : "memory");
        if (k < c0) {
          double s0 = 0.0, s1 = 0.0;
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            if (j < nb) {
              const double2 a = *reinterpret_cast<const double2 *>(u + c0 + j);
              s0 = fma(a.x, xs[c0 + j], s0);
              s1 = fma(a.y, xs[c0 + j + 1], s1);
            }
          }
          y = fma(-rd, s0 + s1, y);
        }
      }
      if (tid < kQuadNbr) {
        double *o = w.wt + static_cast<int64_t>(t_lo + it) * kQuadNbr + tid;
        *o = __dmul_rn(xs[tid], *o);
      }
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------- 5. scatter --
__global__ void quad_count_kernel(int64_t m, QuadWs w) {
  const int64_t g = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (g < m) atomicAdd(w.count + w.nni[g], 1);
}

// exclusive scan of count[0..n) into count[0..n], one CTA
__global__ void __launch_bounds__(1024) quad_scan_kernel(int n, QuadWs w) {
  __shared__ int part[32];
  __shared__ int carry;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < n; base += 1024) {
    const int i = base + tid;
    const int v = i < n ? w.count[i] : 0;
    int incl = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    if (lane == 31) part[warp] = incl;
    __syncthreads();
    int before = carry;
    for (int w2 = 0; w2 < warp; ++w2) before += part[w2];
    if (i < n) w.count[i] = before + incl - v;
    __syncthreads();
    if (tid == 1023) carry = before + incl;
    __syncthreads();
  }
  if (tid == 0) w.count[n] = carry;
}

__global__ void quad_fill_kernel(int64_t m, QuadWs w) {
  const int64_t g = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (g >= m) return;
  const int node = w.nni[g];
  const int pos = w.count[node] + atomicAdd(w.cursor + node, 1);
  w.entry[pos] = static_cast<int32_t>(g);
}

// Per node: its entries in (triangle, slot) order, summed in that order, one
// warp per node.  The order is found by counting, in shared memory: an
// entry's place is the number of smaller ones.  A node has about 160 entries
// (80 neighbours x two triangles per node); a node with more than the staged
// kSumMax sorts its list in place, one lane inserting.  (That insertion sort,
// a thread per node, for all nodes: 850-900 us at 1442 and at 12252 nodes;
// by counting 15 and 57 us.)
constexpr int kSumMax = 512;
constexpr int kSumWarps = 4;

__global__ void __launch_bounds__(32 * kSumWarps) quad_sum_kernel(int n, QuadWs w, double *__restrict__ weights) {
  __shared__ int32_t s_e[kSumWarps][kSumMax];
  __shared__ double s_v[kSumWarps][kSumMax];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = blockIdx.x * kSumWarps + warp;
  if (i >= n) return;
  const int b = w.count[i], e = w.count[i + 1], m = e - b;
  double s = 0.0;
  if (m <= kSumMax) {
    int32_t *se = s_e[warp];
    double *sv = s_v[warp];
    for (int k = lane; k < m; k += 32) se[k] = w.entry[b + k];
    __syncwarp();
    for (int k = lane; k < m; k += 32) {
      const int32_t v = se[k];
      int at = 0;
      for (int q = 0; q < m; ++q) at += se[q] < v;
      sv[at] = w.wt[v];
    }
    __syncwarp();
    if (lane == 0)
      for (int k = 0; k < m; ++k) s = __dadd_rn(s, sv[k]);
  } else if (lane == 0) {
    int32_t *en = w.entry;
    for (int p = b + 1; p < e; ++p) {
      const int32_t v = en[p];
      int q = p - 1;
      while (q >= b && en[q] > v) {
        en[q + 1] = en[q];
        --q;
      }
      en[q + 1] = v;
    }
    for (int p = b; p < e; ++p) s = __dadd_rn(s, w.wt[en[p]]);
  }
  if (lane == 0) weights[i] = s;
}

// The systems go through in chunks, so that their records stay within 72 MB.
constexpr int64_t kTriChunk = 32768;

static int hash_bits(int64_t ntri) {
  int b = 6;
  while ((1ll << b) < 4 * ntri) ++b;
  return b;
}

static size_t quad_layout(int64_t n, int64_t ntri, QuadWs *w, char *base) {
  const int hb = hash_bits(ntri);
  const int64_t H = 1ll << hb;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off = round_up(off + bytes, 256);
    return base ? base + o : nullptr;
  };
  QuadWs q{};
  q.tri = reinterpret_cast<int32_t *>(take(sizeof(int32_t) * 3 * ntri));
  q.tnorm = reinterpret_cast<double *>(take(sizeof(double) * 3 * ntri));
  q.mid = reinterpret_cast<double *>(take(sizeof(double) * 3 * ntri));
  q.enorm = reinterpret_cast<double *>(take(sizeof(double) * 9 * ntri));
  q.hkey = reinterpret_cast<long long *>(take(sizeof(long long) * H));
  q.hid = reinterpret_cast<int32_t *>(take(sizeof(int32_t) * 2 * H));
  q.nni = reinterpret_cast<int32_t *>(take(sizeof(int32_t) * kQuadNbr * ntri));
  q.wt = reinterpret_cast<double *>(take(sizeof(double) * kQuadNbr * ntri));
  q.rec = reinterpret_cast<double *>(take(sizeof(double) * kTriRec * std::min(ntri, kTriChunk)));
  q.count = reinterpret_cast<int32_t *>(take(sizeof(int32_t) * (n + 1)));
  q.cursor = reinterpret_cast<int32_t *>(take(sizeof(int32_t) * n));
  q.entry = reinterpret_cast<int32_t *>(take(sizeof(int32_t) * kQuadNbr * ntri));
  q.hbits = hb;
  if (w) *w = q;
  return off;
}

}  // namespace f3d

extern "C" {

int f3d_surface_quadrature_workspace_bytes(int64_t n, int64_t ntri, size_t *bytes) {
  if (!bytes) return F3D_ERR_NULL;
  if (n < 0 || ntri < 0) return F3D_ERR_SHAPE;
  if (n > f3d::kQuadMaxNodes) return F3D_ERR_TOO_LARGE;
  *bytes = f3d::quad_layout(n, ntri, nullptr, nullptr);
  return F3D_OK;
}

int f3d_surface_quadrature(const double *nodes, int64_t n, const int32_t *triangles, int64_t ntri,
                           const double *gradient, double *weights, int32_t *neighbors, void *workspace,
                           size_t workspace_bytes, void *stream) {
  if (n < f3d::kQuadNbr || ntri < 1 || ntri > (1ll << 24)) return F3D_ERR_SHAPE;
  if (n > f3d::kQuadMaxNodes) return F3D_ERR_TOO_LARGE;
  if (!nodes || !triangles || !gradient || !weights || !workspace) return F3D_ERR_NULL;
  if (!f3d::aligned(nodes, 8) || !f3d::aligned(gradient, 8) || !f3d::aligned(weights, 8) ||
      !f3d::aligned(workspace, 256) || !f3d::aligned(triangles, 4) || (neighbors && !f3d::aligned(neighbors, 4)))
    return F3D_ERR_ALIGN;
  f3d::QuadWs w{};
  const size_t need = f3d::quad_layout(n, ntri, &w, static_cast<char *>(workspace));
  if (workspace_bytes < need) return F3D_ERR_WORKSPACE;
  if (neighbors) w.nni = neighbors;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int *err = f3d::device_error_word();
  const int64_t H = 1ll << w.hbits;
  if (cudaMemsetAsync(w.hkey, 0xff, sizeof(long long) * H, st) != cudaSuccess ||
      cudaMemsetAsync(w.hid, 0xff, sizeof(int32_t) * 2 * H, st) != cudaSuccess ||
      cudaMemsetAsync(w.count, 0, sizeof(int32_t) * (n + 1), st) != cudaSuccess ||
      cudaMemsetAsync(w.cursor, 0, sizeof(int32_t) * n, st) != cudaSuccess)
    return F3D_ERR_CUDA;
  const int nt = static_cast<int>(ntri), nn = static_cast<int>(n);
  f3d::quad_prep_kernel<<<(nt + 127) / 128, 128, 0, st>>>(nodes, nn, triangles, nt, w, err);
  f3d::quad_edges_kernel<<<(3 * nt + 127) / 128, 128, 0, st>>>(nn, nt, w, err);
  const int tile = static_cast<int>(std::min<int64_t>(n, f3d::kKnnTile));
  const size_t knn_smem = 2 * (sizeof(double) * (f3d::kQuadNbr + f3d::kKnnCand) +
                               sizeof(int) * (f3d::kKnnCand + f3d::kQuadNbr)) +
                          sizeof(int) * f3d::kKnnBins + 2 * sizeof(unsigned) * ((tile + f3d::kQuadNbr + 3) & ~3);
  // the opt-in limit counts the kernel's static shared memory too: ask for
  // what this call needs
  static size_t attr_bytes[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return F3D_ERR_CUDA;
  if (knn_smem > attr_bytes[dev]) {
    if (cudaFuncSetAttribute(f3d::quad_knn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(knn_smem)) != cudaSuccess)
      return F3D_ERR_CUDA;
    attr_bytes[dev] = knn_smem;
  }
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f3d::quad_knn_kernel, f3d::kKnnThreads, knn_smem) !=
          cudaSuccess ||
      per_sm < 1)
    return F3D_ERR_CUDA;
  const int64_t knn_grid = std::min<int64_t>((ntri + 1) / 2, static_cast<int64_t>(per_sm) * f3d::sm_count());
  f3d::quad_knn_kernel<<<static_cast<unsigned>(knn_grid), f3d::kKnnThreads, knn_smem, st>>>(nodes, nn, w.mid, nt,
                                                                                            tile, w.nni, err);
  static bool tri_attr[64] = {false};
  if (!tri_attr[dev]) {
    if (cudaFuncSetAttribute(f3d::quad_triangle_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(f3d::kTriSmem)) != cudaSuccess)
      return F3D_ERR_CUDA;
    tri_attr[dev] = true;
  }
  for (int64_t lo = 0; lo < ntri; lo += f3d::kTriChunk) {
    const int count = static_cast<int>(std::min(ntri - lo, f3d::kTriChunk));
    f3d::quad_geometry_kernel<<<count, f3d::kGeoThreads, 0, st>>>(nodes, gradient, static_cast<int>(lo), w);
    const int grid = std::min(count, 2 * f3d::sm_count());
    f3d::quad_triangle_kernel<<<grid, f3d::kTriThreads, f3d::kTriSmem, st>>>(static_cast<int>(lo), count, w, err);
  }
  const int64_t m = f3d::kQuadNbr * ntri;
  f3d::quad_count_kernel<<<static_cast<unsigned>((m + 255) / 256), 256, 0, st>>>(m, w);
  f3d::quad_scan_kernel<<<1, 1024, 0, st>>>(nn, w);
  f3d::quad_fill_kernel<<<static_cast<unsigned>((m + 255) / 256), 256, 0, st>>>(m, w);
  f3d::quad_sum_kernel<<<(nn + f3d::kSumWarps - 1) / f3d::kSumWarps, 32 * f3d::kSumWarps, 0, st>>>(nn, w, weights);
  return f3d::launch_status();
}

}  // extern "C"
