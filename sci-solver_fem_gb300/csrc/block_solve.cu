// block_solve.cu -- several right-hand sides with one hierarchy, solved together.
//
// The columns are taken in blocks of kBlock = 8.  Inside a block every column runs its
// own flexible PCG (CG_Flex_Cycle, cgcycle.cu:6-69, the method of the single-column
// solve) with its own step lengths, but the eight advance in lockstep and every operator
// application is a sparse matrix times an n x 8 block (SpMM): the FP64 outer operator,
// each level's in-partition and cross-partition entries, R and P are read once per block
// instead of once per column, and the coarsest solve X = A_c^{-1} B is a dense FP64
// product on the tensor cores (DMMA, mma.sync m8n8k4 f64).  A column that has converged
// keeps its x and r (its step length is zero) while the others go on.  Block vectors are
// row-major n x 8, so one gather of a column index fetches the row's eight values in one
// 32-byte (FP32) or 64-byte (FP64) access.
//
// The smoother is the partition-block weighted Jacobi of the single-column V-cycle
// (gauss_seidel.cu:1278-1376, 3626-3736) on the same groups of partitions, with row sums
// in entry order; the V-cycle is AMG_Level::cycle (amg_level.cu:22-71).
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "context.cuh"

namespace femgpu {

namespace {

constexpr int kBlock = 8;
constexpr int kBG = 608;   // fixed reduction grid (4 x 152 SMs) x kBT threads
constexpr int kBT = 256;
constexpr unsigned kAll = 0xffffffffu;

// per-column scalar slots: slot s of column j is sc[s * kBlock + j]
enum BSlot { B_BN = 0, B_NR, B_PY, B_ALPHA, B_RZ, B_RZNEW, B_ZROLD, B_BETA, B_ACTIVE, B_ITS, B_FLAG, B_NSLOT };
// block-wide slots after the per-column ones
enum BGlobal { G_FIRST = B_NSLOT * kBlock, G_IT, G_TOL, G_MAXIT, G_ANY, G_FLEX, G_COUNT };

template <class T>
struct V8 {
  T v[kBlock];
};

template <class T>
__device__ __forceinline__ V8<T> ld8(const T* p) {
  V8<T> r;
  if constexpr (sizeof(T) == 4) {
    const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
    r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
  } else {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const double2 a = reinterpret_cast<const double2*>(p)[q];
      r.v[2 * q] = a.x;
      r.v[2 * q + 1] = a.y;
    }
  }
  return r;
}

template <class T>
__device__ __forceinline__ void st8(T* p, const V8<T>& r) {
  if constexpr (sizeof(T) == 4) {
    reinterpret_cast<float4*>(p)[0] = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(r.v[4], r.v[5], r.v[6], r.v[7]);
  } else {
#pragma unroll
    for (int q = 0; q < 4; q++) reinterpret_cast<double2*>(p)[q] = make_double2(r.v[2 * q], r.v[2 * q + 1]);
  }
}

// ---- vector kernels and reductions over the fixed grid -------------------------------
// A block vector is walked as n x 4 pairs of columns, pair q mod 4 = columns 2 (q mod 4) and
// the next: consecutive threads read consecutive 16 bytes, and a thread keeps its two columns
// because the grid's stride is a multiple of 4.  (A thread per row, 64 bytes apart, ran these
// kernels at 0.8 TB/s: 64^3, eight columns, dot 67 -> 22 us, update 66 -> 26 us.)
constexpr int kPairs = kBlock / 2;

// Block sums of a pair of columns per thread (the pair of threadIdx.x mod 4) to
// out[0 .. 8), by threads 0..7.
__device__ __forceinline__ void block_columns(double2 v, double (*sh)[kBlock], double* out) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o >= kPairs; o >>= 1) {
    v.x += __shfl_xor_sync(kAll, v.x, o);
    v.y += __shfl_xor_sync(kAll, v.y, o);
  }
  __syncthreads();  // sh may still be read from an earlier call
  if (lane < kPairs) {
    sh[w][2 * lane] = v.x;
    sh[w][2 * lane + 1] = v.y;
  }
  __syncthreads();
  if (threadIdx.x < kBlock) {
    double t = sh[0][threadIdx.x];
    for (int q = 1; q < kBT / 32; q++) t += sh[q][threadIdx.x];
    out[threadIdx.x] = t;
  }
}

// After every block wrote its partials: true in the block that finishes last.
__device__ __forceinline__ bool last_block(unsigned* counter) {
  __shared__ bool s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(counter, 1u) == gridDim.x - 1;
  __syncthreads();
  if (s_last) __threadfence();
  return s_last;
}

// Total of partial[b * 8 + j] over b for column j = threadIdx.x mod 8, in a fixed order; in
// threads 0..7.
__device__ __forceinline__ double column_total(const double* partial, double (*sh)[kBlock]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, j = threadIdx.x & (kBlock - 1);
  double s = 0.0;
#pragma unroll 4
  for (int b = threadIdx.x / kBlock; b < kBG; b += kBT / kBlock) s += partial[b * kBlock + j];
  s += __shfl_xor_sync(kAll, s, 8);
  s += __shfl_xor_sync(kAll, s, 16);
  __syncthreads();
  if (lane < kBlock) sh[w][lane] = s;
  __syncthreads();
  s = sh[0][j];
  for (int q = 1; q < kBT / 32; q++) s += sh[q][j];
  return s;
}

// ---- FP64 outer kernels -------------------------------------------------------------
// out (n x 8, permuted order) from the caller's column-major B (column j at B + j * ldb)
__global__ void blk_in_kernel(int n, int kc, const int32_t* __restrict__ perm, const double* __restrict__ B,
                              int64_t ldb, double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  V8<double> r;
#pragma unroll
  for (int j = 0; j < kBlock; j++) r.v[j] = j < kc ? B[j * ldb + i] : 0.0;
  st8(out + (int64_t)perm[i] * kBlock, r);
}

__global__ void blk_out_kernel(int n, int kc, const int32_t* __restrict__ perm, const double* __restrict__ in,
                               double* __restrict__ X, int64_t ldx) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const V8<double> r = ld8(in + (int64_t)perm[i] * kBlock);
#pragma unroll
  for (int j = 0; j < kBlock; j++)
    if (j < kc) X[j * ldx + i] = r.v[j];
}

// sc[slot] = a.b per column (and sc[slot2] = a.c when c != nullptr).
__global__ void __launch_bounds__(kBT) blk_dot_kernel(int n, const double* __restrict__ a,
                                                       const double* __restrict__ b, const double* __restrict__ c,
                                                       double* partial, double* sc, int slot, int slot2,
                                                       unsigned* counter) {
  __shared__ double sh[kBT / 32][kBlock];
  const double2 *va = reinterpret_cast<const double2*>(a), *vb = reinterpret_cast<const double2*>(b),
                *vc = reinterpret_cast<const double2*>(c);
  const int64_t pairs = (int64_t)n * kPairs;
  double2 s1 = make_double2(0.0, 0.0), s2 = s1;
#pragma unroll 2
  for (int64_t q = (int64_t)blockIdx.x * kBT + threadIdx.x; q < pairs; q += (int64_t)kBG * kBT) {
    const double2 x = va[q], y = vb[q];
    s1.x = fma(x.x, y.x, s1.x);
    s1.y = fma(x.y, y.y, s1.y);
    if (c) {
      const double2 z = vc[q];
      s2.x = fma(x.x, z.x, s2.x);
      s2.y = fma(x.y, z.y, s2.y);
    }
  }
  block_columns(s1, sh, partial + blockIdx.x * kBlock);
  if (c) block_columns(s2, sh, partial + (kBG + blockIdx.x) * kBlock);
  if (!last_block(counter)) return;
  const double t1 = column_total(partial, sh);
  if (threadIdx.x < kBlock) sc[slot * kBlock + threadIdx.x] = t1;
  if (c) {
    const double t2 = column_total(partial + kBG * kBlock, sh);
    if (threadIdx.x < kBlock) sc[slot2 * kBlock + threadIdx.x] = t2;
  }
  if (threadIdx.x == 0) *counter = 0u;
}

// Columns 2 t, 2 t + 1 (t = the lane's pair) of row i of the outer FP64 operator times the
// block (sliced layout when off != nullptr: rows 32 s .. 32 s + 31 column-major from off[s],
// padding column -1; else CSR), entries in order, four in flight.  Four lanes share a row, so
// a gathered row of the block is one 64-byte access.  Bound by the FP64 pipe: 8 fused
// multiply-adds per entry (64^3: 32 M, 64 us at 0.5 T/s).
__device__ __forceinline__ double2 outer_row(int i, int t, const int32_t* __restrict__ off,
                                             const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                                             const double* __restrict__ v, const double* __restrict__ p) {
  const double2* __restrict__ p2 = reinterpret_cast<const double2*>(p);
  double2 s = make_double2(0.0, 0.0);
  const int end = off ? off[(i >> 5) + 1] : rp[i + 1];
  const int step = off ? 32 : 1;
  for (int e = off ? off[i >> 5] + (i & 31) : rp[i]; e < end; e += 4 * step) {
    int c[4];
    double a[4];
    double2 x[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      c[k] = e + k * step < end ? ci[e + k * step] : -1;
      a[k] = e + k * step < end ? v[e + k * step] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) x[k] = c[k] >= 0 ? p2[(int64_t)c[k] * kPairs + t] : make_double2(0.0, 0.0);
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (c[k] >= 0) {
        s.x = fma(a[k], x[k].x, s.x);
        s.y = fma(a[k], x[k].y, s.y);
      }
  }
  return s;
}

// y = A p, p.y per column; the last block forms alpha = rz / p.y for the active columns
// (a non-positive or non-finite p.y flags the column and stops it).  64^3, eight columns:
// 105 -> 84 us (a thread per row, eight columns each).
__global__ void __launch_bounds__(kBT) blk_spmv_dot_kernel(int n, const int32_t* __restrict__ off,
                                                            const int32_t* __restrict__ rp,
                                                            const int32_t* __restrict__ ci,
                                                            const double* __restrict__ v,
                                                            const double* __restrict__ p, double* __restrict__ y,
                                                            double* partial, double* sc, unsigned* counter) {
  __shared__ double sh[kBT / 32][kBlock];
  const double2* p2 = reinterpret_cast<const double2*>(p);
  double2* y2 = reinterpret_cast<double2*>(y);
  const int64_t pairs = (int64_t)n * kPairs;
  double2 acc = make_double2(0.0, 0.0);
  for (int64_t q = (int64_t)blockIdx.x * kBT + threadIdx.x; q < pairs; q += (int64_t)kBG * kBT) {
    const double2 s = outer_row((int)(q / kPairs), (int)(q & (kPairs - 1)), off, rp, ci, v, p), pi = p2[q];
    y2[q] = s;
    acc.x = fma(s.x, pi.x, acc.x);
    acc.y = fma(s.y, pi.y, acc.y);
  }
  block_columns(acc, sh, partial + blockIdx.x * kBlock);
  if (!last_block(counter)) return;
  const double t = column_total(partial, sh);
  const int j = threadIdx.x;
  if (j < kBlock) {
    double* s = sc;
    s[B_PY * kBlock + j] = t;
    double alpha = 0.0;
    if (s[B_ACTIVE * kBlock + j] != 0.0) {
      if (t > 0.0 && isfinite(t)) {
        alpha = s[B_RZ * kBlock + j] / t;
      } else {
        s[B_FLAG * kBlock + j] = 1.0;
        s[B_ACTIVE * kBlock + j] = 0.0;
      }
    }
    s[B_ALPHA * kBlock + j] = alpha;
  }
  if (j == 0) *counter = 0u;
}

// y = A x (start of the solve).
__global__ void blk_spmv_kernel(int n, const int32_t* __restrict__ off, const int32_t* __restrict__ rp,
                                const int32_t* __restrict__ ci, const double* __restrict__ v,
                                const double* __restrict__ x, double* __restrict__ y) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q < (int64_t)n * kPairs)
    reinterpret_cast<double2*>(y)[q] = outer_row((int)(q / kPairs), (int)(q & (kPairs - 1)), off, rp, ci, v, x);
}

// r = b - y
__global__ void blk_sub_kernel(int n, const double* __restrict__ b, const double* __restrict__ y,
                               double* __restrict__ r) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= (int64_t)n * kPairs) return;
  const double2 vb = reinterpret_cast<const double2*>(b)[q], vy = reinterpret_cast<const double2*>(y)[q];
  reinterpret_cast<double2*>(r)[q] = make_double2(vb.x - vy.x, vb.y - vy.y);
}

// beta per column (cgcycle.cu:52-54; Polak-Ribiere when flexible), 0 on the first
// iteration and for stopped columns; rz = rz_new.
__global__ void blk_beta_kernel(double* sc) {
  const int j = threadIdx.x;
  if (j >= kBlock) return;
  const bool first = sc[G_FIRST] != 0.0, flex = sc[G_FLEX] != 0.0;
  const double rz = sc[B_RZ * kBlock + j], rzn = sc[B_RZNEW * kBlock + j];
  double beta = 0.0;
  if (!first && sc[B_ACTIVE * kBlock + j] != 0.0) beta = flex ? (rzn - sc[B_ZROLD * kBlock + j]) / rz : rzn / rz;
  sc[B_BETA * kBlock + j] = beta;
  sc[B_RZ * kBlock + j] = rzn;
  __syncwarp(0xffu);
  if (j == 0) sc[G_FIRST] = 0.0;
}

// p = z + beta p
__global__ void blk_pupdate_kernel(int n, const double* __restrict__ sc, const double* __restrict__ z,
                                   double* __restrict__ p) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= (int64_t)n * kPairs) return;
  const double2 beta = reinterpret_cast<const double2*>(sc + B_BETA * kBlock)[q & (kPairs - 1)];
  const double2 vz = reinterpret_cast<const double2*>(z)[q], vp = reinterpret_cast<const double2*>(p)[q];
  reinterpret_cast<double2*>(p)[q] = make_double2(fma(beta.x, vp.x, vz.x), fma(beta.y, vp.y, vz.y));
}

// x += alpha p; r -= alpha y (rold = r first when flexible); r.r per column; the last
// block advances the iteration count and stops converged, broken or exhausted columns.
__global__ void __launch_bounds__(kBT) blk_update_kernel(int n, double* sc, const double* __restrict__ p,
                                                          const double* __restrict__ y, double* __restrict__ x,
                                                          double* __restrict__ r, double* __restrict__ rold,
                                                          double* partial, unsigned* counter) {
  __shared__ double sh[kBT / 32][kBlock];
  const double2 alpha = reinterpret_cast<const double2*>(sc + B_ALPHA * kBlock)[threadIdx.x & (kPairs - 1)];
  const double2 *vp = reinterpret_cast<const double2*>(p), *vy = reinterpret_cast<const double2*>(y);
  double2 *vx = reinterpret_cast<double2*>(x), *vr = reinterpret_cast<double2*>(r), *vo = reinterpret_cast<double2*>(rold);
  const int64_t pairs = (int64_t)n * kPairs;
  double2 acc = make_double2(0.0, 0.0);
#pragma unroll 2
  for (int64_t q = (int64_t)blockIdx.x * kBT + threadIdx.x; q < pairs; q += (int64_t)kBG * kBT) {
    const double2 rr = vr[q], pp = vp[q], xx = vx[q], yy = vy[q];
    if (rold) vo[q] = rr;
    vx[q] = make_double2(fma(alpha.x, pp.x, xx.x), fma(alpha.y, pp.y, xx.y));
    const double2 nr = make_double2(fma(-alpha.x, yy.x, rr.x), fma(-alpha.y, yy.y, rr.y));
    vr[q] = nr;
    acc.x = fma(nr.x, nr.x, acc.x);
    acc.y = fma(nr.y, nr.y, acc.y);
  }
  block_columns(acc, sh, partial + blockIdx.x * kBlock);
  if (!last_block(counter)) return;
  const double t = column_total(partial, sh);
  __shared__ int s_any;
  if (threadIdx.x == 0) s_any = 0;
  __syncthreads();
  const int j = threadIdx.x;
  const double it = sc[G_IT] + 1.0;
  if (j < kBlock) {
    sc[B_NR * kBlock + j] = t;
    if (sc[B_ACTIVE * kBlock + j] != 0.0) {
      sc[B_ITS * kBlock + j] = it;
      const double bn = sqrt(sc[B_BN * kBlock + j]);
      const double nr = sqrt(t);
      if (!isfinite(nr)) {
        sc[B_FLAG * kBlock + j] = 1.0;
        sc[B_ACTIVE * kBlock + j] = 0.0;
      } else if (nr / (bn > 0.0 ? bn : 1.0) <= sc[G_TOL]) {
        sc[B_ACTIVE * kBlock + j] = 0.0;
      } else {
        s_any = 1;
      }
    }
  }
  __syncthreads();
  if (j == 0) {
    sc[G_IT] = it;
    sc[G_ANY] = (s_any && it < sc[G_MAXIT]) ? 1.0 : 0.0;
    *counter = 0u;
  }
}

// ---- V-cycle kernels (hierarchy precision T) ------------------------------------------------
// C neighbouring columns of a block row.
template <class T, int C>
struct __align__(C * sizeof(T)) Cols {
  T v[C];
};
template <class T>
using Pair = Cols<T, 2>;

// An in-partition entry in shared memory: its value and the byte offset of the x row it reads.
template <class T>
struct __align__(2 * sizeof(T)) BlkEntry {
  T v;
  int off;
};

template <class T>
__global__ void blk_cast_in_kernel(int64_t m, const double* __restrict__ in, T* __restrict__ out) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q < m) out[q] = (T)in[q];
}

template <class T>
__global__ void blk_cast_out_kernel(int64_t m, const T* __restrict__ in, double* __restrict__ out) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q < m) out[q] = (double)in[q];
}

template <class T>
__device__ __forceinline__ T relax1(T x, T b, T sax, T d, T dinv, T w) {
  T t = b - sax;
  t = t - d * x;
  return x + (w * t) * dinv;
}

// Partition-block weighted Jacobi on one group of consecutive partitions (rows
// [grows[g], grows[g + 1]), at most kBlkRows of them) and C LPR of the eight columns per CTA:
// LPR lanes per row with C columns each, times EL lanes that share the row's entries, and up
// to LPR EL rows per thread.  The group's x is double-buffered in shared memory, its
// in-partition entries are staged there once (eight loads in flight); a row's bounds,
// diagonal, right-hand side and x stay in registers.  Pre (POST == false): x0 = w b / d,
// `inner` sweeps, then x and r = b - A_in x - d x; with b64 the right-hand side is read in
// FP64, rounded, and kept in b_store for the post relax.  Post: b - A_out x_in, `inner` sweeps
// from x_in; with z64 the result is written there in FP64.  With EL = 1 row sums run in entry
// order, else lane j adds entries j, j + EL, ... and the lanes' sums are added by shuffles.
// Bound by shared-memory instructions and their latency on full levels, by staging and
// barriers on small ones.  64^3, pre relaxes of the levels of 708, 32 and 2 groups:
// 95 -> 68, 65 -> 25, 85 -> 27 us (before: all eight columns by one thread per row, bounds
// and diagonal from global memory in every sweep).
constexpr int kBlkRows = 512;
constexpr int kBlkThreads = 512;

template <class T, bool POST, int C, int LPR, int EL>
__global__ void __launch_bounds__(kBlkThreads, sizeof(T) == 4 ? 2 : 1) blk_smooth_kernel(
    const int32_t* __restrict__ grows, const int32_t* __restrict__ irp, const int32_t* __restrict__ ici,
    const T* __restrict__ iv, const int32_t* __restrict__ orp, const int32_t* __restrict__ oci,
    const T* __restrict__ ov, const T* __restrict__ diag, const T* __restrict__ dinv, const T* __restrict__ b,
    const double* __restrict__ b64, T* __restrict__ b_store, T w, int inner, const T* __restrict__ x_in,
    T* __restrict__ x_out, double* __restrict__ z64, T* __restrict__ r_out, int mcap) {
  using V = Cols<T, C>;
  constexpr int SPLIT = kBlock / (C * LPR);  // CTAs per group
  constexpr int RV = kBlock / C;             // vectors per block row in global memory
  constexpr int RP = LPR * EL;               // rows per thread, lanes per row
  constexpr int RB = C * LPR * sizeof(T);    // bytes of a row of x in shared memory
  extern __shared__ __align__(16) unsigned char sm[];
  unsigned char* const x0b = sm;
  unsigned char* const x1b = sm + (size_t)mcap * RB;
  BlkEntry<T>* const ent = reinterpret_cast<BlkEntry<T>*>(x1b + (size_t)mcap * RB);
  const int g = blockIdx.x / SPLIT;
  const int rs = grows[g], m = grows[g + 1] - rs;
  const int es = irp[rs], ne = irp[rs + m] - es;
  const int per = blockDim.x / RP, lr = threadIdx.x / RP;
  const int lp = threadIdx.x % LPR, el = (threadIdx.x / LPR) % EL;
  const int vec = (blockIdx.x % SPLIT) * LPR + lp;  // of the row's vectors in global memory
  for (int q0 = threadIdx.x; q0 < ne; q0 += 8 * blockDim.x) {
    T v[8];
    int c[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int q = q0 + k * blockDim.x;
      v[k] = q < ne ? iv[es + q] : (T)0;
      c[k] = q < ne ? ici[es + q] : 0;
    }
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int q = q0 + k * blockDim.x;
      if (q < ne) {
        BlkEntry<T> e;
        e.v = v[k];
        e.off = (c[k] - rs) * RB;
        ent[q] = e;
      }
    }
  }
  const V* xin = reinterpret_cast<const V*>(x_in);
  V x[RP], bb[RP];
  T d[RP], di[RP];
  int e0[RP], e1[RP];
#pragma unroll
  for (int u = 0; u < RP; u++) {
    const int t = u * per + lr, row = rs + t;
    const bool live = t < m;
    e0[u] = e1[u] = 0;
    d[u] = di[u] = (T)1;
#pragma unroll
    for (int k = 0; k < C; k++) x[u].v[k] = bb[u].v[k] = (T)0;
    const int64_t at = (int64_t)row * RV + vec;
    int o0 = 0, o1 = 0;
    if (live) {
      e0[u] = irp[row] - es;
      e1[u] = irp[row + 1] - es;
      d[u] = diag[row];
      di[u] = dinv[row];
      if (!POST && b64) {
        const Cols<double, 2>* src = reinterpret_cast<const Cols<double, 2>*>(b64 + at * C);
#pragma unroll
        for (int k = 0; k < C / 2; k++) {
          const Cols<double, 2> v = src[k];
          bb[u].v[2 * k] = (T)v.v[0];
          bb[u].v[2 * k + 1] = (T)v.v[1];
        }
        if (el == 0) reinterpret_cast<V*>(b_store)[at] = bb[u];
      } else {
        bb[u] = reinterpret_cast<const V*>(b)[at];
      }
      if (POST) {
        x[u] = xin[at];
        o0 = orp[row];
        o1 = orp[row + 1];
      } else {
#pragma unroll
        for (int k = 0; k < C; k++) x[u].v[k] = (w * bb[u].v[k]) * di[u];
      }
    }
    if (POST) {
      V so;  // EL > 1: this lane's share of A_out x
#pragma unroll
      for (int k = 0; k < C; k++) so.v[k] = (T)0;
      for (int o = o0 + el; o < o1; o += 4 * EL) {
        int c[4];
        T a[4];
        V xo[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          c[q] = o + q * EL < o1 ? oci[o + q * EL] : row;
          a[q] = o + q * EL < o1 ? ov[o + q * EL] : (T)0;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) xo[q] = xin[(int64_t)c[q] * RV + vec];
#pragma unroll
        for (int q = 0; q < 4; q++)
          if (o + q * EL < o1) {
#pragma unroll
            for (int k = 0; k < C; k++) {
              if (EL == 1) bb[u].v[k] = bb[u].v[k] - a[q] * xo[q].v[k];
              else so.v[k] = fma(a[q], xo[q].v[k], so.v[k]);
            }
          }
      }
      if (EL > 1) {
#pragma unroll
        for (int k = 0; k < C; k++) {
#pragma unroll
          for (int f = LPR; f < RP; f <<= 1) so.v[k] = so.v[k] + __shfl_xor_sync(kAll, so.v[k], f);
          bb[u].v[k] = bb[u].v[k] - so.v[k];
        }
      }
    }
    if (live && el == 0) reinterpret_cast<V*>(x0b + (size_t)t * RB)[lp] = x[u];
  }
  __syncthreads();
  // every lane of the warp calls it (with EL > 1 the lanes' sums are exchanged)
  auto row_sum = [&](const unsigned char* cur, int a, int z) {
    const unsigned char* base = cur + lp * sizeof(V);
    V s;
#pragma unroll
    for (int k = 0; k < C; k++) s.v[k] = (T)0;
    int e = a + el;
    for (; e + EL < z; e += 2 * EL) {
      const BlkEntry<T> p = ent[e], q = ent[e + EL];
      const V xp = *reinterpret_cast<const V*>(base + p.off), xq = *reinterpret_cast<const V*>(base + q.off);
#pragma unroll
      for (int k = 0; k < C; k++) s.v[k] = fma(p.v, xp.v[k], s.v[k]);
#pragma unroll
      for (int k = 0; k < C; k++) s.v[k] = fma(q.v, xq.v[k], s.v[k]);
    }
    if (e < z) {
      const BlkEntry<T> p = ent[e];
      const V xp = *reinterpret_cast<const V*>(base + p.off);
#pragma unroll
      for (int k = 0; k < C; k++) s.v[k] = fma(p.v, xp.v[k], s.v[k]);
    }
    if (EL > 1) {
#pragma unroll
      for (int k = 0; k < C; k++)
#pragma unroll
        for (int f = LPR; f < RP; f <<= 1) s.v[k] = s.v[k] + __shfl_xor_sync(kAll, s.v[k], f);
    }
    return s;
  };
  unsigned char* cur = x0b;
  unsigned char* nxt = x1b;
  for (int it = 0; it < inner; it++) {
#pragma unroll
    for (int u = 0; u < RP; u++) {
      const int t = u * per + lr;
      const V s = row_sum(cur, e0[u], e1[u]);
#pragma unroll
      for (int k = 0; k < C; k++) x[u].v[k] = relax1(x[u].v[k], bb[u].v[k], s.v[k], d[u], di[u], w);
      if (t < m && el == 0) reinterpret_cast<V*>(nxt + (size_t)t * RB)[lp] = x[u];
    }
    __syncthreads();
    unsigned char* tmp = cur;
    cur = nxt;
    nxt = tmp;
  }
#pragma unroll
  for (int u = 0; u < RP; u++) {
    const int t = u * per + lr;
    const int64_t at = (int64_t)(rs + t) * RV + vec;
    const bool mine = t < m && el == 0;
    if (mine) {
      if (POST && z64) {
#pragma unroll
        for (int k = 0; k < C / 2; k++) {
          Cols<double, 2> z;
          z.v[0] = (double)x[u].v[2 * k];
          z.v[1] = (double)x[u].v[2 * k + 1];
          reinterpret_cast<Cols<double, 2>*>(z64 + at * C)[k] = z;
        }
      } else {
        reinterpret_cast<V*>(x_out)[at] = x[u];
      }
    }
    if (!POST) {
      const V s = row_sum(cur, e0[u], e1[u]);
      V r;
#pragma unroll
      for (int k = 0; k < C; k++) r.v[k] = (bb[u].v[k] - s.v[k]) - d[u] * x[u].v[k];
      if (mine) reinterpret_cast<V*>(r_out)[at] = r;
    }
  }
}

// The same relaxes for groups that blk_smooth_kernel does not take (more than kBlkRows rows,
// or entries that do not fit beside x): one CTA per group, a thread per row with all eight
// columns, the entries read from global memory in every sweep.
template <class T, bool POST>
__global__ void __launch_bounds__(512) blk_smooth_large_kernel(
    const int32_t* __restrict__ grows, const int32_t* __restrict__ irp, const int32_t* __restrict__ ici,
    const T* __restrict__ iv, const int32_t* __restrict__ orp, const int32_t* __restrict__ oci,
    const T* __restrict__ ov, const T* __restrict__ diag, const T* __restrict__ dinv, const T* __restrict__ b,
    const double* __restrict__ b64, T* __restrict__ b_store, T w, int inner, const T* __restrict__ x_in,
    T* __restrict__ x_out, double* __restrict__ z64, T* __restrict__ r_out, int mcap) {
  extern __shared__ __align__(16) unsigned char sm[];
  T* xa = reinterpret_cast<T*>(sm);
  T* xb = xa + (int64_t)mcap * kBlock;
  T* sb = xb + (int64_t)mcap * kBlock;
  const int rs = grows[blockIdx.x], m = grows[blockIdx.x + 1] - rs;
  for (int t = threadIdx.x; t < m; t += blockDim.x) {
    const int row = rs + t;
    V8<T> bb, x0;
    if (!POST && b64) {
      const V8<double> v = ld8(b64 + (int64_t)row * kBlock);
#pragma unroll
      for (int j = 0; j < kBlock; j++) bb.v[j] = (T)v.v[j];
      st8(b_store + (int64_t)row * kBlock, bb);
    } else {
      bb = ld8(b + (int64_t)row * kBlock);
    }
    if (POST) {
      x0 = ld8(x_in + (int64_t)row * kBlock);
      for (int e = orp[row]; e < orp[row + 1]; e++) {
        const T a = ov[e];
        const V8<T> xo = ld8(x_in + (int64_t)oci[e] * kBlock);
#pragma unroll
        for (int j = 0; j < kBlock; j++) bb.v[j] = bb.v[j] - a * xo.v[j];
      }
    } else {
      const T di = dinv[row];
#pragma unroll
      for (int j = 0; j < kBlock; j++) x0.v[j] = (w * bb.v[j]) * di;
    }
    st8(sb + (int64_t)t * kBlock, bb);
    st8(xa + (int64_t)t * kBlock, x0);
  }
  __syncthreads();
  auto row_sum = [&](const T* cur, int row) {
    V8<T> s;
#pragma unroll
    for (int j = 0; j < kBlock; j++) s.v[j] = (T)0;
    for (int e = irp[row]; e < irp[row + 1]; e++) {
      const T a = iv[e];
      const V8<T> xv = ld8(cur + (int64_t)(ici[e] - rs) * kBlock);
#pragma unroll
      for (int j = 0; j < kBlock; j++) s.v[j] = fma(a, xv.v[j], s.v[j]);
    }
    return s;
  };
  T* cur = xa;
  T* nxt = xb;
  for (int it = 0; it < inner; it++) {
    for (int t = threadIdx.x; t < m; t += blockDim.x) {
      const int row = rs + t;
      const V8<T> s = row_sum(cur, row), xc = ld8(cur + (int64_t)t * kBlock), bb = ld8(sb + (int64_t)t * kBlock);
      const T d = diag[row], di = dinv[row];
      V8<T> xn;
#pragma unroll
      for (int j = 0; j < kBlock; j++) xn.v[j] = relax1(xc.v[j], bb.v[j], s.v[j], d, di, w);
      st8(nxt + (int64_t)t * kBlock, xn);
    }
    __syncthreads();
    T* tmp = cur;
    cur = nxt;
    nxt = tmp;
  }
  for (int t = threadIdx.x; t < m; t += blockDim.x) {
    const int row = rs + t;
    const V8<T> xc = ld8(cur + (int64_t)t * kBlock);
    if (POST && z64) {
      V8<double> z;
#pragma unroll
      for (int j = 0; j < kBlock; j++) z.v[j] = (double)xc.v[j];
      st8(z64 + (int64_t)row * kBlock, z);
    } else {
      st8(x_out + (int64_t)row * kBlock, xc);
    }
    if (!POST) {
      const V8<T> s = row_sum(cur, row), bb = ld8(sb + (int64_t)t * kBlock);
      const T d = diag[row];
      V8<T> r;
#pragma unroll
      for (int j = 0; j < kBlock; j++) r.v[j] = (bb.v[j] - s.v[j]) - d * xc.v[j];
      st8(r_out + (int64_t)row * kBlock, r);
    }
  }
}

// M x on the block: y = M x (restriction), y += M x (prolongation) or y -= M x (the
// cross-partition part of the residual, preAout_kernel, gauss_seidel.cu:1977-2015).  Four
// lanes share a row's eight columns and G such quadruples its entries (every G-th, four in
// flight); the quadruples' sums are added by shuffles.  G grows with the average row
// (spmm_groups): a thread per row left the restrictions, rows of 26 to 250 entries on few
// rows, without parallelism.  64^3, restrictions of levels 0, 1, 2: 82 -> 13, 147 -> 15,
// 83 -> 12 us.
enum SpmmMode { SPMM_SET, SPMM_ADD, SPMM_SUB };

template <class T, int MODE, int G>
__global__ void __launch_bounds__(128) blk_spmm_kernel(int n, const int32_t* __restrict__ rp,
                                                       const int32_t* __restrict__ ci, const T* __restrict__ v,
                                                       const T* __restrict__ x, T* __restrict__ y) {
  constexpr int LANES = kPairs * G;
  const int i = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / LANES);
  const int t = threadIdx.x & (kPairs - 1), gr = (threadIdx.x / kPairs) & (G - 1);
  const bool live = i < n;
  const Pair<T>* x2 = reinterpret_cast<const Pair<T>*>(x);
  Pair<T> s;
  s.v[0] = s.v[1] = (T)0;
  const int e1 = live ? rp[i + 1] : 0;
  for (int e = live ? rp[i] + gr : 0; e < e1; e += 4 * G) {
    int c[4];
    T a[4];
    Pair<T> xv[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      c[k] = e + k * G < e1 ? ci[e + k * G] : -1;
      a[k] = e + k * G < e1 ? v[e + k * G] : (T)0;
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (c[k] >= 0) xv[k] = x2[(int64_t)c[k] * kPairs + t];
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (c[k] >= 0) {
        s.v[0] = fma(a[k], xv[k].v[0], s.v[0]);
        s.v[1] = fma(a[k], xv[k].v[1], s.v[1]);
      }
  }
#pragma unroll
  for (int o = kPairs; o < LANES; o <<= 1) {
    s.v[0] = s.v[0] + __shfl_xor_sync(kAll, s.v[0], o);
    s.v[1] = s.v[1] + __shfl_xor_sync(kAll, s.v[1], o);
  }
  if (!live || gr != 0) return;
  Pair<T>* out = reinterpret_cast<Pair<T>*>(y) + (int64_t)i * kPairs + t;
  if (MODE != SPMM_SET) {
    const Pair<T> o = *out;
    s.v[0] = MODE == SPMM_ADD ? o.v[0] + s.v[0] : o.v[0] - s.v[0];
    s.v[1] = MODE == SPMM_ADD ? o.v[1] + s.v[1] : o.v[1] - s.v[1];
  }
  *out = s;
}

// Coarsest level, X = Ainv B for the eight columns on the FP64 tensor cores: warp w forms
// rows 8w .. 8w + 7 of X with mma.sync m8n8k4 f64 steps over the inner dimension (A tile =
// 8 x 4 of the explicit inverse, row-major; B tile = 4 x 8 of the block).  Rows and inner
// indices past n are zero.
template <class T>
__global__ void blk_coarse_kernel(int n, const double* __restrict__ inv, const T* __restrict__ b,
                                  T* __restrict__ x) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int r0 = w * 8;
  if (r0 >= n) return;  // the whole warp
  double d0 = 0.0, d1 = 0.0;
  const int arow = r0 + (lane >> 2), acol = lane & 3;  // A fragment: (lane / 4, lane % 4)
  const int brow = lane & 3, bcol = lane >> 2;         // B fragment: (lane % 4, lane / 4)
  for (int k0 = 0; k0 < n; k0 += 4) {
    const double a = (arow < n && k0 + acol < n) ? inv[(int64_t)arow * n + k0 + acol] : 0.0;
    const double bv = (k0 + brow < n) ? (double)b[(int64_t)(k0 + brow) * kBlock + bcol] : 0.0;
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(bv));
  }
  const int crow = r0 + (lane >> 2), ccol = (lane & 3) * 2;  // D fragment: (lane / 4, 2 (lane % 4) + i)
  if (crow < n) {
    x[(int64_t)crow * kBlock + ccol] = (T)d0;
    x[(int64_t)crow * kBlock + ccol + 1] = (T)d1;
  }
}

// ---- per-handle state -----------------------------------------------------------------------
template <class T>
struct BlockLevel {
  DBuf<T> b, x, r, xo, t;
};

template <class T>
struct BlockState : BlockStateBase {
  uint64_t gen = ~0ull;
  std::vector<BlockLevel<T>> lv;
  DBuf<double> vb, vx, vr, vz, vp, vy, vrold, part, sc;
  DBuf<unsigned> cnt;
  double* h_sc = nullptr;
  // the block PCG loop captured as a CUDA graph (conditional while node), per flexible flag
  cudaGraphExec_t exec[2] = {nullptr, nullptr};
  int64_t nodes[2] = {0, 0};
  ~BlockState() override {
    for (cudaGraphExec_t e : exec)
      if (e) cudaGraphExecDestroy(e);
    if (h_sc) cudaFreeHost(h_sc);
  }
};

// Continue the device-side block loop while a column is still running.
__global__ void blk_check_kernel(const double* sc, cudaGraphConditionalHandle loop) {
  cudaGraphSetConditional(loop, sc[G_ANY] != 0.0 ? 1u : 0u);
}

// Shared memory of blk_smooth_large_kernel: x twice and the right-hand side (m x 8 each).
template <class T>
size_t blk_large_smem(int mcap) {
  return (size_t)mcap * kBlock * sizeof(T) * 3;
}

// Shared memory of blk_smooth_kernel for `cols` columns: x twice and the staged entries.
template <class T>
size_t blk_smooth_smem(const Level<T>& L, int cols) {
  return (size_t)L.max_group_rows * cols * sizeof(T) * 2 + (size_t)L.max_group_ents * sizeof(BlkEntry<T>);
}

// Columns per CTA of blk_smooth_kernel: all eight while the groups fill the SMs twice over,
// two otherwise (four CTAs per group); 0 when the level's groups do not fit it.
// 64^3, level of 32 groups, pre relax: 65 us with all eight columns in a CTA (before), 35 us
// with two, 25 us with two and four lanes per row's entries.
constexpr size_t kBlockStageLimit = 200 * 1024;
template <class T>
int blk_columns(const Level<T>& L) {
  if (L.max_group_rows > kBlkRows) return 0;
  if (L.ngroups >= 2 * 152 && blk_smooth_smem(L, kBlock) <= (sizeof(T) == 4 ? kBlockStageLimit / 2 : kBlockStageLimit))
    return kBlock;
  return blk_smooth_smem(L, 2) <= kBlockStageLimit ? 2 : 0;
}

template <class T, bool POST, int C, int LPR, int EL>
void launch_blk_smooth_as(cudaStream_t s, const Level<T>& L, const T* b, const double* b64, T* b_store, T w, int inner,
                          const T* x_in, T* x_out, double* z64, T* r_out) {
  const int thr = std::min(kBlkThreads, (L.max_group_rows * LPR * EL + 31) / 32 * 32);
  const size_t smem = blk_smooth_smem(L, C * LPR);
  ensure_smem(blk_smooth_kernel<T, POST, C, LPR, EL>, smem);
  FG_LAUNCH((blk_smooth_kernel<T, POST, C, LPR, EL>), L.ngroups * (kBlock / (C * LPR)), thr, smem, s, L.grows.p,
            L.Ain.rp.p, L.Ain.ci.p, L.Ain.v.p, L.Aout.rp.p, L.Aout.ci.p, L.Aout.v.p, L.diag.p, L.dinv.p, b, b64,
            b_store, w, inner, x_in, x_out, z64, r_out, L.max_group_rows);
}

template <class T, bool POST>
void launch_blk_smooth(cudaStream_t s, const Level<T>& L, const T* b, const double* b64, T* b_store, T w, int inner,
                       const T* x_in, T* x_out, double* z64, T* r_out) {
  constexpr int C = 16 / (int)sizeof(T);  // 16-byte reads of x
  const int cols = blk_columns(L);
  if (cols == kBlock) {
    launch_blk_smooth_as<T, POST, C, kBlock / C, 1>(s, L, b, b64, b_store, w, inner, x_in, x_out, z64, r_out);
    return;
  }
  if (cols == 2) {
    // rows of 16 entries and more are shared by four lanes
    if (L.Ain.nnz >= 16 * (int64_t)L.n)
      launch_blk_smooth_as<T, POST, 2, 1, 4>(s, L, b, b64, b_store, w, inner, x_in, x_out, z64, r_out);
    else
      launch_blk_smooth_as<T, POST, 2, 1, 1>(s, L, b, b64, b_store, w, inner, x_in, x_out, z64, r_out);
    return;
  }
  const int thr = std::min(512, std::max(32, (L.max_group_rows + 31) / 32 * 32));
  const size_t smem = blk_large_smem<T>(L.max_group_rows);
  ensure_smem(blk_smooth_large_kernel<T, POST>, smem);
  FG_LAUNCH((blk_smooth_large_kernel<T, POST>), L.ngroups, thr, smem, s, L.grows.p, L.Ain.rp.p, L.Ain.ci.p, L.Ain.v.p,
            L.Aout.rp.p, L.Aout.ci.p, L.Aout.v.p, L.diag.p, L.dinv.p, b, b64, b_store, w, inner, x_in, x_out, z64,
            r_out, L.max_group_rows);
}

// Quadruples of lanes per row of blk_spmm_kernel: each takes about eight entries of an
// average row (two rounds of its four loads in flight).
template <class T>
int spmm_groups(const DCsr<T>& M) {
  const double avg = M.n > 0 ? (double)M.nnz / M.n : 0.0;
  return avg <= 8.0 ? 1 : avg <= 16.0 ? 2 : avg <= 32.0 ? 4 : 8;
}

template <class T, int MODE>
void launch_blk_spmm(cudaStream_t s, const DCsr<T>& M, const T* x, T* y) {
  const int G = spmm_groups(M);
  const int g = grid_for((int64_t)M.n * kPairs * G, 128);
#define FG_SPMM(GG) FG_LAUNCH((blk_spmm_kernel<T, MODE, GG>), g, 128, 0, s, M.n, M.rp.p, M.ci.p, M.v.p, x, y)
  switch (G) {
    case 1: FG_SPMM(1); break;
    case 2: FG_SPMM(2); break;
    case 4: FG_SPMM(4); break;
    default: FG_SPMM(8); break;
  }
#undef FG_SPMM
}

// b_in -> x_out; at level 0 with r64 the right-hand side is read from r64 in FP64 (and its
// rounded copy kept in b_in), with z64 the result goes there in FP64.
template <class T>
void block_vcycle(Ctx& c, Hierarchy<T>& H, BlockState<T>& S, int l, T* b_in, T* x_out, const double* r64 = nullptr,
                  double* z64 = nullptr) {
  cudaStream_t s = c.stream;
  Level<T>& L = *H.L[l];
  const int n = L.A.n;
  if (L.coarsest) {
    FG_LAUNCH(blk_coarse_kernel<T>, grid_for((int64_t)((n + 7) / 8) * 32, 128), 128, 0, s, n, L.Ainv.p, b_in, x_out);
    return;
  }
  BlockLevel<T>& W = S.lv[l];
  const T w = (T)c.cfg.smootherWeight;
  // pre relax: x, r = b - A_in x - d x, then r -= A_out x
  launch_blk_smooth<T, false>(s, L, b_in, r64, b_in, w, c.cfg.preInnerIters, (const T*)nullptr, W.x.p,
                              (double*)nullptr, W.r.p);
  launch_blk_spmm<T, SPMM_SUB>(s, L.Aout, W.x.p, W.r.p);
  BlockLevel<T>& NW = S.lv[l + 1];
  launch_blk_spmm<T, SPMM_SET>(s, L.R, W.r.p, NW.t.p);
  block_vcycle(c, H, S, l + 1, NW.t.p, NW.xo.p);
  launch_blk_spmm<T, SPMM_ADD>(s, L.P, NW.xo.p, W.x.p);
  T* src = W.x.p;
  for (int rl = 0; rl < c.cfg.postRelaxes; rl++) {
    const bool last = rl + 1 == c.cfg.postRelaxes;
    T* dst = last ? x_out : (src == W.x.p ? W.r.p : W.x.p);
    launch_blk_smooth<T, true>(s, L, b_in, (const double*)nullptr, (T*)nullptr, w, c.cfg.postInnerIters, src, dst,
                               last ? z64 : (double*)nullptr, (T*)nullptr);
    src = dst;
  }
  if (c.cfg.postRelaxes == 0) {
    if (z64)
      FG_LAUNCH(blk_cast_out_kernel<T>, grid_for((int64_t)n * kBlock, 256), 256, 0, s, (int64_t)n * kBlock, W.x.p, z64);
    else
      FG_CUDA(cudaMemcpyAsync(x_out, W.x.p, (size_t)n * kBlock * sizeof(T), cudaMemcpyDeviceToDevice, s));
  }
}

template <class T>
BlockState<T>& block_state(Ctx& c, Hierarchy<T>& H) {
  BlockState<T>* S = dynamic_cast<BlockState<T>*>(c.block.get());
  if (!S || S->gen != c.hier_gen) {
    auto fresh = std::make_unique<BlockState<T>>();
    S = fresh.get();
    c.block = std::move(fresh);
    cudaStream_t s = c.stream;
    const int64_t n = c.A.n;
    for (int l = 0; l < H.num_levels; l++) {
      const Level<T>& L = *H.L[l];
      BlockLevel<T> W;
      const int64_t m = (int64_t)L.A.n * kBlock;
      W.b.alloc(m, s);
      W.x.alloc(m, s);
      W.xo.alloc(m, s);
      W.t.alloc(m, s);
      if (!L.coarsest) {
        W.r.alloc(m, s);
        const size_t smem = blk_large_smem<T>(L.max_group_rows);
        FG_REQUIRE(smem <= 227 * 1024, FEMGPU_ERR_LIMIT,
                   "a smoother group is too large for the multi-right-hand-side smoother's shared memory");
      }
      S->lv.push_back(std::move(W));
    }
    for (DBuf<double>* v : {&S->vb, &S->vx, &S->vr, &S->vz, &S->vp, &S->vy, &S->vrold}) v->alloc(n * kBlock, s);
    S->part.alloc((size_t)2 * kBlock * kBG, s);
    S->sc.alloc(G_COUNT, s);
    S->cnt.alloc(4, s);
    S->cnt.zero();
    FG_CUDA(cudaMallocHost((void**)&S->h_sc, G_COUNT * sizeof(double)));
    S->gen = c.hier_gen;
  }
  return *S;
}

// z = M r for the block (permuted level-0 FP64 vectors).
template <class T>
void block_precondition(Ctx& c, Hierarchy<T>& H, BlockState<T>& S, const double* r, double* z) {
  cudaStream_t s = c.stream;
  const int64_t m = (int64_t)H.L[0]->A.n * kBlock;
  BlockLevel<T>& W = S.lv[0];
  if constexpr (std::is_same<T, double>::value) {
    block_vcycle(c, H, S, 0, const_cast<double*>(r), z);  // the V-cycle only reads its input
  } else if (H.L[0]->coarsest) {
    FG_LAUNCH(blk_cast_in_kernel<T>, grid_for(m, 256), 256, 0, s, m, r, W.b.p);
    block_vcycle(c, H, S, 0, W.b.p, W.xo.p);
    FG_LAUNCH(blk_cast_out_kernel<T>, grid_for(m, 256), 256, 0, s, m, W.xo.p, z);
  } else {
    block_vcycle(c, H, S, 0, W.b.p, W.xo.p, r, z);  // level 0 reads r and writes z itself
  }
}

template <class T>
void block_solve_columns(Ctx& c, Hierarchy<T>& H, int kc, const double* B, int64_t ldb, double* X, int64_t ldx,
                         int* iters, double* relres, femgpu_status* status) {
  cudaStream_t s = c.stream;
  BlockState<T>& S = block_state(c, H);
  const int n = c.A.n;
  const int32_t* off = c.sliced ? c.s_off.p : nullptr;
  const int32_t* rp = c.sliced ? nullptr : c.A0p.rp.p;
  const int32_t* ci = c.sliced ? c.s_ci.p : c.A0p.ci.p;
  const double* v = c.sliced ? c.s_v.p : c.A0p.v.p;
  double* sc = S.sc.p;
  double* part = S.part.p;
  const int flexible = c.cfg.flexibleCG;
  FG_LAUNCH(blk_in_kernel, grid_for(n, 256), 256, 0, s, n, kc, c.perm0.p, B, ldb, S.vb.p);
  FG_LAUNCH(blk_in_kernel, grid_for(n, 256), 256, 0, s, n, kc, c.perm0.p, X, ldx, S.vx.p);
  // scalars: b.b, r = b - A x, r.r, active columns
  FG_CUDA(cudaMemsetAsync(sc, 0, G_COUNT * sizeof(double), s));
  FG_CUDA(cudaMemsetAsync(S.cnt.p, 0, S.cnt.n * sizeof(unsigned), s));
  FG_CUDA(cudaMemsetAsync(S.vp.p, 0, S.vp.n * sizeof(double), s));
  FG_LAUNCH(blk_dot_kernel, kBG, kBT, 0, s, n, S.vb.p, S.vb.p, (const double*)nullptr, part, sc, (int)B_BN, 0,
            S.cnt.p);
  FG_LAUNCH(blk_spmv_kernel, grid_for((int64_t)n * kPairs, 256), 256, 0, s, n, off, rp, ci, v, S.vx.p, S.vy.p);
  FG_LAUNCH(blk_sub_kernel, grid_for((int64_t)n * kPairs, 256), 256, 0, s, n, S.vb.p, S.vy.p, S.vr.p);
  FG_LAUNCH(blk_dot_kernel, kBG, kBT, 0, s, n, S.vr.p, S.vr.p, (const double*)nullptr, part, sc, (int)B_NR, 0,
            S.cnt.p);
  FG_CUDA(cudaMemcpyAsync(S.h_sc, sc, G_COUNT * sizeof(double), cudaMemcpyDeviceToHost, s));
  FG_CUDA(cudaStreamSynchronize(s));
  double* h = S.h_sc;
  const double tol = c.cfg.tolerance;
  bool any = false;
  for (int j = 0; j < kBlock; j++) {
    const double bn = sqrt(h[B_BN * kBlock + j]);
    const bool act = j < kc && !(sqrt(h[B_NR * kBlock + j]) / (bn > 0.0 ? bn : 1.0) <= tol);
    h[B_ACTIVE * kBlock + j] = act ? 1.0 : 0.0;
    any = any || act;
  }
  h[G_FIRST] = 1.0;
  h[G_IT] = 0.0;
  h[G_TOL] = tol;
  h[G_MAXIT] = (double)c.cfg.maxIters;
  h[G_FLEX] = flexible ? 1.0 : 0.0;
  h[G_ANY] = (any && c.cfg.maxIters > 0) ? 1.0 : 0.0;
  FG_CUDA(cudaMemcpyAsync(sc, h, G_COUNT * sizeof(double), cudaMemcpyHostToDevice, s));
  // one block PCG iteration (the last kernel decides whether another one runs)
  auto iteration = [&]() {
    block_precondition(c, H, S, S.vr.p, S.vz.p);
    FG_LAUNCH(blk_dot_kernel, kBG, kBT, 0, s, n, S.vz.p, S.vr.p, flexible ? (const double*)S.vrold.p : nullptr, part,
              sc, (int)B_RZNEW, (int)B_ZROLD, S.cnt.p);
    FG_LAUNCH(blk_beta_kernel, 1, kBlock, 0, s, sc);
    FG_LAUNCH(blk_pupdate_kernel, grid_for((int64_t)n * kPairs, 256), 256, 0, s, n, sc, S.vz.p, S.vp.p);
    FG_LAUNCH(blk_spmv_dot_kernel, kBG, kBT, 0, s, n, off, rp, ci, v, S.vp.p, S.vy.p, part, sc, S.cnt.p + 1);
    FG_LAUNCH(blk_update_kernel, kBG, kBT, 0, s, n, sc, S.vp.p, S.vy.p, S.vx.p, S.vr.p,
              flexible ? S.vrold.p : nullptr, part, S.cnt.p + 2);
  };
  if (h[G_ANY] != 0.0) {
    // the iterations run on the device as a CUDA graph with a conditional while node,
    // captured once per hierarchy (FEMGPU_HOST_LOOP: launched one by one from the host)
    cudaGraphExec_t& exec = S.exec[flexible ? 1 : 0];
    if (!exec && !getenv("FEMGPU_HOST_LOOP")) {
      const int64_t before = g_kernel_launches.load();
      cudaGraph_t g = nullptr;
      bool ok = cudaGraphCreate(&g, 0) == cudaSuccess;
      cudaGraphConditionalHandle loop;
      cudaGraphNodeParams cp = {};
      if (ok) ok = cudaGraphConditionalHandleCreate(&loop, g, 1, cudaGraphCondAssignDefault) == cudaSuccess;
      if (ok) {
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = loop;
        cp.conditional.type = cudaGraphCondTypeWhile;
        cp.conditional.size = 1;
        cudaGraphNode_t node;
        ok = cudaGraphAddNode(&node, g, nullptr, nullptr, 0, &cp) == cudaSuccess;
      }
      if (ok)
        ok = cudaStreamBeginCaptureToGraph(s, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                           cudaStreamCaptureModeThreadLocal) == cudaSuccess;
      if (ok) {
        try {
          iteration();
          FG_LAUNCH(blk_check_kernel, 1, 1, 0, s, sc, loop);
        } catch (...) {
          ok = false;
        }
        cudaGraph_t captured = nullptr;
        ok = cudaStreamEndCapture(s, &captured) == cudaSuccess && ok;
      }
      if (ok) ok = cudaGraphInstantiate(&exec, g, 0) == cudaSuccess;
      if (!ok) {
        (void)cudaGetLastError();
        exec = nullptr;
      }
      if (g) cudaGraphDestroy(g);
      S.nodes[flexible ? 1 : 0] = g_kernel_launches.load() - before;
      g_kernel_launches.store(before);  // counted per iteration after each run
    }
    if (exec) {
      FG_CUDA(cudaGraphLaunch(exec, s));
      FG_CUDA(cudaMemcpyAsync(h, sc, G_COUNT * sizeof(double), cudaMemcpyDeviceToHost, s));
      FG_CUDA(cudaStreamSynchronize(s));
      g_kernel_launches.fetch_add(S.nodes[flexible ? 1 : 0] * (int64_t)h[G_IT]);
    } else {
      while (h[G_ANY] != 0.0) {
        iteration();
        FG_CUDA(cudaMemcpyAsync(h, sc, G_COUNT * sizeof(double), cudaMemcpyDeviceToHost, s));
        FG_CUDA(cudaStreamSynchronize(s));
      }
    }
  }
  FG_LAUNCH(blk_out_kernel, grid_for(n, 256), 256, 0, s, n, kc, c.perm0.p, S.vx.p, X, ldx);
  for (int j = 0; j < kc; j++) {
    const double bn = sqrt(h[B_BN * kBlock + j]);
    const double rr = sqrt(h[B_NR * kBlock + j]) / (bn > 0.0 ? bn : 1.0);
    iters[j] = (int)h[B_ITS * kBlock + j];
    relres[j] = rr;
    status[j] = (h[B_FLAG * kBlock + j] != 0.0 || !std::isfinite(rr)) ? FEMGPU_ERR_BREAKDOWN
                : rr <= tol                                              ? FEMGPU_OK
                                                                         : FEMGPU_ERR_NOT_CONVERGED;
  }
}

}  // namespace

void block_solve_device(Ctx& c, int nrhs, const double* d_B, int64_t ldb, double* d_X, int64_t ldx, int* iters,
                        double* relres, femgpu_status* status) {
  FG_REQUIRE(c.has_hierarchy, FEMGPU_ERR_NOT_READY, "call femgpu_setup first");
  for (int j0 = 0; j0 < nrhs; j0 += kBlock) {
    const int kc = std::min(kBlock, nrhs - j0);
    if (c.cfg.precision == 1)
      block_solve_columns(c, static_cast<Hierarchy<double>&>(*c.H), kc, d_B + j0 * ldb, ldb, d_X + j0 * ldx, ldx,
                          iters + j0, relres + j0, status + j0);
    else
      block_solve_columns(c, static_cast<Hierarchy<float>&>(*c.H), kc, d_B + j0 * ldb, ldb, d_X + j0 * ldx, ldx,
                          iters + j0, relres + j0, status + j0);
  }
}

}  // namespace femgpu
