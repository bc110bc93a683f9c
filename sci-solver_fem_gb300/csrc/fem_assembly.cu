// fem_assembly.cu -- mesh pattern and P1 element assembly on the device.
//
// Pattern: vertex -> (element, local vertex) incidence lists, sorted, then each
// row's column set is the sorted union of the vertices of its incident elements
// (the row of tetmesh2ell / trimesh2ell, src/core/cuda/cutil.cu:168-230,297-348,
// with the diagonal in its sorted place).
//
// Assembly: one thread per element computes the element's matrix
// (perform_element_loop_3D.cuh:480-627 / perform_element_loop_2D.cuh:287-372) and stores
// its rows as 32-byte sectors; one thread per row of the operator then gathers its
// entries from the incident elements in element order.  No floating-point atomics: the sum at
// every slot is taken in element order, so results are bitwise reproducible and
// equal to a sequential element loop.  Tetrahedra use a fused multiply-add gradient
// formulation (tet_gradients), within a few units in the last place of the reference's
// cofactor inverse; triangles follow the reference's arithmetic.
#include "context.cuh"
#include "quadrature.h"

namespace femgpu {

namespace {

__constant__ double c_tet_mass[10];
// Triangle quadrature: wx[6], wy[6], (1 - zx)[6], (1 + zx)[6], (1 - zy)[6], (1 + zy)[6]
__constant__ double c_tri_q[36];

// Row r of an element matrix is one 32-byte sector of the element table (four doubles,
// the last one unused for triangles), at 4 * (e * k + r): the incidence code of the row's
// vertex, so the gather reads exactly the sectors it adds.
__device__ __forceinline__ void st_row(double* p, double a, double b, double c, double d) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

// x / D rounded to nearest, for D = 6, 12, 20, in three FP64 operations (the compiler's
// division takes about three times as many, and these kernels are bound by the FP64 pipe:
// GB300 issues 2 per SM and clock).  With y = RN(1 / D) the quotient q = RN(x y) is within
// 1.2 ulp of x / D, so x - D q is exact, and q + (x - D q) y is off x / D by less than
// 2^-52 ulp before its rounding.  x / D is never that near a rounding boundary: in units of
// ulp(q), x is a multiple of 4 (D = 6), 8 (12) or 16 (20) and a boundary lies at an odd
// multiple of D / 2, so they differ by at least 1 / D ulp (Brisebarre, Muller and Raina,
// "Accelerating correctly rounded floating-point division when the divisor is known in
// advance", IEEE Trans. Computers 2004).  Tiny, huge and special x take the division.
template <int D>
__device__ __forceinline__ double div_const(double x) {
  static_assert(D == 6 || D == 12 || D == 20, "proved for these divisors");
  constexpr double y = 1.0 / D;
  const unsigned hi = (unsigned)__double2hiint(x) & 0x7fffffffu;
  if (hi - 0x03000000u >= 0x7a000000u) return x / (double)D;
  const double q = x * y;
  return fma(fma(-(double)D, q, x), y, q);
}

__device__ __forceinline__ double label_coef(int label) {
  // co of element_loop_3d_kernel (perform_element_loop_3D.cuh:585-612)
  return label == 2 ? 2.0 : label == 3 ? 3.0 : label == 4 ? 4.0 : label == 5 ? 5.0 : label == 6 ? 6.0 : 1.0;
}

// ---- pattern ----------------------------------------------------------------------
__global__ void incidence_count_kernel(const int32_t* conn, int64_t nslots, int32_t* deg, int nv, int32_t* bad) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < nslots; q += (int64_t)gridDim.x * blockDim.x) {
    int v = conn[q];
    if (v < 0 || v >= nv) {
      atomicExch(bad, 1);
      continue;
    }
    atomicAdd(&deg[v], 1);
  }
}

__global__ void incidence_fill_kernel(const int32_t* conn, int64_t nslots, const int32_t* vstart, int32_t* cursor,
                                      int32_t* inc) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < nslots; q += (int64_t)gridDim.x * blockDim.x) {
    int v = conn[q];
    int pos = atomicAdd(&cursor[v], 1);
    inc[vstart[v] + pos] = (int32_t)q;  // q = e * k + a
  }
}

__global__ void times_k_kernel(const int32_t* deg, int nv, int k, int32_t* out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += gridDim.x * blockDim.x) out[i] = deg[i] * k;
}

__global__ void candidates_kernel(const int32_t* conn, const int32_t* vstart, const int32_t* inc, const int32_t* coff,
                                  int nv, int k, int32_t* cand) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
    int o = coff[v];
    for (int q = vstart[v]; q < vstart[v + 1]; q++) {
      int e = inc[q] / k;
      for (int b = 0; b < k; b++) cand[o++] = conn[(int64_t)e * k + b];
    }
  }
}

__global__ void compact_rows_kernel(const int32_t* cand, const int32_t* coff, const int32_t* rowptr, int nv,
                                    int32_t* cols) {
  // warp per row
  int lane = threadIdx.x & 31;
  for (int v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < nv; v += (gridDim.x * blockDim.x) >> 5) {
    int len = rowptr[v + 1] - rowptr[v];
    for (int t = lane; t < len; t += 32) cols[rowptr[v] + t] = cand[coff[v] + t];
  }
}

__global__ void graph_from_pattern_kernel(const int32_t* rowptr, const int32_t* cols, int n, int32_t* xadj,
                                          int32_t* adj) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int o = rowptr[i] - i;  // one diagonal entry per earlier row
    if (i == 0) xadj[0] = 0;
    int c = 0;
    for (int e = rowptr[i]; e < rowptr[i + 1]; e++)
      if (cols[e] != i) adj[o + c++] = cols[e];
    xadj[i + 1] = o + c;
  }
}

// ---- assembly --------------------------------------------------------------------
// P1 basis gradients of tetrahedron e from its edge vectors (a fused multiply-add
// formulation; the CPU oracle evaluates the same operations in the same order):
// with a = p1 - p0, b = p2 - p0, c = p3 - p0 and det = a . (b x c),
// grad l1 = (b x c) / det, grad l2 = (c x a) / det, grad l3 = (a x b) / det,
// grad l0 = -((grad l1 + grad l2) + grad l3); the volume is |det| / 6.  About a quarter of
// the floating-point work of the 4x4 cofactor inverse (perform_element_loop_3D.cuh:
// 525-583), which it matches to a few units in the last place.
__device__ __forceinline__ void cross_fma(const double u[3], const double v[3], double w[3]) {
  w[0] = fma(u[1], v[2], -(u[2] * v[1]));
  w[1] = fma(u[2], v[0], -(u[0] * v[2]));
  w[2] = fma(u[0], v[1], -(u[1] * v[0]));
}

__device__ __forceinline__ void tet_gradients(const double* __restrict__ xyz, const int32_t* __restrict__ conn,
                                              int64_t e, double& det, double g[4][3]) {
  double p[4][3];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int64_t v = conn[e * 4 + q];
#pragma unroll
    for (int d = 0; d < 3; d++) p[q][d] = xyz[v * 3 + d];
  }
  double a[3], b[3], c[3], bc[3], ca[3], ab[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    a[d] = p[1][d] - p[0][d];
    b[d] = p[2][d] - p[0][d];
    c[d] = p[3][d] - p[0][d];
  }
  cross_fma(b, c, bc);
  cross_fma(c, a, ca);
  cross_fma(a, b, ab);
  det = fma(a[0], bc[0], fma(a[1], bc[1], a[2] * bc[2]));
  const double inv = 1.0 / det;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    g[1][d] = bc[d] * inv;
    g[2][d] = ca[d] * inv;
    g[3][d] = ab[d] * inv;
    g[0][d] = -((g[1][d] + g[2][d]) + g[3][d]);
  }
}

// Element matrices co K_e + lambda M_e of P1 tetrahedra (perform_element_loop_3D.cuh:28-116,
// 480-627): K_ab = vol grad l_a . grad l_b, the mass from the reference-element integrand
// table times |det| / 8.  Bound by the FP64 pipe (about 105 operations per element without
// the mass term, 120 with it).  MASS == false is lambda = 0: the term is then a signed
// zero, which the row sums (they start from +0) do not see.  Entry-major table, a
// division by 6 and the mass term always added: 101^3 cells (6.2 M elements), lambda = 1:
// 1365 us, now 1311; 96^3 cells, lambda = 0: 1172 us, now 909.
template <bool MASS>
__global__ void element3d_kernel(const double* __restrict__ xyz, const int32_t* __restrict__ conn,
                                 const int32_t* __restrict__ labels, const double* __restrict__ coef, int64_t ne,
                                 double lambda, double* __restrict__ ev) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += (int64_t)gridDim.x * blockDim.x) {
    double det, g[4][3];
    tet_gradients(xyz, conn, e, det, g);
    const double co = coef ? coef[e] : (labels ? label_coef(labels[e]) : 1.0);
    const double wk = div_const<6>(fabs(det)) * co;
    const double jac = fabs(det) * 0.125;
    double m[4][4];
    int c = 0;
#pragma unroll
    for (int kk = 0; kk < 4; kk++) {
#pragma unroll
      for (int q = kk; q < 4; q++) {
        const double st = fma(g[kk][0], g[q][0], fma(g[kk][1], g[q][1], g[kk][2] * g[q][2])) * wk;
        m[kk][q] = m[q][kk] = MASS ? fma(lambda, c_tet_mass[c] * jac, st) : st;
        c++;
      }
    }
    double* o = ev + e * 16;
#pragma unroll
    for (int r = 0; r < 4; r++) st_row(o + 4 * r, m[r][0], m[r][1], m[r][2], m[r][3]);
  }
}

// Element matrices of P1 triangles in the reference's arithmetic
// (perform_element_loop_2D.cuh:287-372).  The mass quadrature's basis values at a point do
// not depend on the entry: they are formed once per point for the three basis functions and
// used for all six entries, and everything that depends on one quadrature index alone is
// formed once per index; the operations that remain are the same in the same order (the
// factors 0.5 are exact and are applied where they cost least).  Bound by the FP64 pipe:
// 44 operations per point, 36 points.  500^2 cells (0.5 M elements), lambda = 1: 1798 us
// (every entry its own quadrature: 5139 us).  MASS == false is lambda = 0, as above.
template <bool MASS>
__global__ void __launch_bounds__(128) element2d_kernel(const double* __restrict__ xyz,
                                                        const int32_t* __restrict__ conn,
                                                        const double* __restrict__ coef, int64_t ne, double lambda,
                                                        double* __restrict__ ev) {
  const double *wx = c_tri_q, *wy = c_tri_q + 6, *zxm = c_tri_q + 12, *zxp = c_tri_q + 18, *zym = c_tri_q + 24,
               *zyp = c_tri_q + 30;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += (int64_t)gridDim.x * blockDim.x) {
    double x[3], y[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      int v = conn[e * 3 + a];
      x[a] = xyz[(int64_t)v * 3];
      y[a] = xyz[(int64_t)v * 3 + 1];
    }
    double area = fabs(x[0] * y[2] - x[0] * y[1] + x[1] * y[0] - x[1] * y[2] + x[2] * y[1] - x[2] * y[0]) / 2.0;
    double a11 = x[0], a12 = y[0], a13 = 1.0, a21 = x[1], a22 = y[1], a23 = 1.0, a31 = x[2], a32 = y[2], a33 = 1.0;
    double det = a11 * a22 * a33 + a21 * a32 * a13 + a31 * a12 * a23 - a11 * a32 * a23 - a31 * a22 * a13 - a21 * a12 * a33;
    double cf[9] = {(a22 * a33 - a23 * a32) / det, (a23 * a31 - a21 * a33) / det, (a21 * a32 - a22 * a31) / det,
                    (a13 * a32 - a12 * a33) / det, (a11 * a33 - a13 * a31) / det, (a12 * a31 - a11 * a32) / det,
                    (a12 * a23 - a13 * a22) / det, (a13 * a21 - a11 * a23) / det, (a11 * a22 - a12 * a21) / det};
    double jacobi = (x[0] * y[1] - x[1] * y[0] - x[0] * y[2] + x[2] * y[0] + x[1] * y[2] - x[2] * y[1]) / 8;
    double co = coef ? coef[e] : 1.0;
    double integral[6] = {0, 0, 0, 0, 0, 0};
    if (MASS) {
      double x2[6], y2[6];  // the third vertex's share of a point, by the second index
#pragma unroll
      for (int j = 0; j < 6; j++) {
        x2[j] = x[2] * zyp[j] * 0.5;
        y2[j] = y[2] * zyp[j] * 0.5;
      }
#pragma unroll 1
      for (int i = 0; i < 6; i++) {
        const double x0 = x[0] * zxm[i] * 0.25, x1 = x[1] * zxp[i] * 0.25;
        const double y0 = y[0] * zxm[i] * 0.25, y1 = y[1] * zxp[i] * 0.25;
        double ty[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int j = 0; j < 6; j++) {
          const double px = x0 * zym[j] + x1 * zym[j] + x2[j];
          const double py = y0 * zym[j] + y1 * zym[j] + y2[j];
          double l[3];
#pragma unroll
          for (int k = 0; k < 3; k++) l[k] = cf[3 * k] * px + cf[3 * k + 1] * py + cf[3 * k + 2];
          int c = 0;
#pragma unroll
          for (int k = 0; k < 3; k++)
#pragma unroll
            for (int q = k; q < 3; q++) {
              ty[c] += l[k] * l[q] * jacobi * wy[j];
              c++;
            }
        }
#pragma unroll
        for (int c = 0; c < 6; c++) integral[c] += ty[c] * wx[i];
      }
    }
    double m[3][3];
    int c = 0;
#pragma unroll
    for (int k = 0; k < 3; k++)
#pragma unroll
      for (int q = k; q < 3; q++) {
        const double st = (cf[3 * k] * cf[3 * q] + cf[3 * k + 1] * cf[3 * q + 1]) * area * co;
        m[k][q] = m[q][k] = MASS ? st + lambda * integral[c] : st;
        c++;
      }
    double* o = ev + e * 12;
#pragma unroll
    for (int r = 0; r < 3; r++) st_row(o + 4 * r, m[r][0], m[r][1], m[r][2], 0.0);
  }
}

// Positions within its row of every (incidence, element vertex) pair, for the gather
// below (one binary search each, once per mesh).  An element that names a vertex more than
// once has several entries at one position; the second, third and fourth of them carry their
// turn in the upper two bits, and *repeats is set.
constexpr int kSlotTurn = 6;  // positions are below kSlotRowMax
static_assert(kSlotRowMax <= 1 << kSlotTurn, "turns share a byte with the positions");

__global__ void slot_map_kernel(const int32_t* __restrict__ rowptr, const int32_t* __restrict__ cols,
                                const int32_t* __restrict__ vstart, const int32_t* __restrict__ inc,
                                const int32_t* __restrict__ conn, int nv, int k, uint8_t* __restrict__ slot,
                                int32_t* bad, int32_t* repeats) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
    const int rb = rowptr[v], re = rowptr[v + 1];
    for (int q = vstart[v]; q < vstart[v + 1]; q++) {
      const int e = inc[q] / k;
      int seen[3] = {-1, -1, -1};
      for (int b = 0; b < k; b++) {
        const int col = conn[(int64_t)e * k + b];
        const int s = lower_bound_i32(cols, rb, re, col);
        if (s >= re || cols[s] != col) {
          atomicExch(bad, 1);
          slot[(int64_t)q * k + b] = 0;
          continue;
        }
        int turn = 0;  // earlier vertices of the element that are the same
#pragma unroll
        for (int o = 0; o < 3; o++) {
          turn += o < b && seen[o] == col;
          if (o == b) seen[o] = col;
        }
        if (turn) *repeats = 1;
        slot[(int64_t)q * k + b] = (uint8_t)((s - rb) | turn << kSlotTurn);
      }
    }
  }
}

// Four lanes per row with the row's sums in shared memory (at most kSlotRowMax entries,
// kSlotRowMax + 1 doubles apart per row): lane b adds entry b of each incident element's
// row, in element order, at the position the slot map gives.  The lanes of a row never meet
// in a mesh whose elements have distinct vertices; with REPEATS lanes at one position add one
// after the other, in the order of the element's vertices (such an element's volume is only
// nearly zero after rounding, so its entries are finite).  Bound by the chain of shared-memory
// adds, 24 per row of a tetrahedral mesh, so a row's lanes work side by side and the sectors,
// codes and slots of the next four elements are loaded ahead.  101^3 cells: 335 us (one thread per row,
// entry-major table, four 8-byte reads of as many sectors per incidence: 874 us; one thread
// per row on this table: 705 us).
constexpr int kGatherThreads = 256;

template <int K, bool REPEATS>
__global__ void __launch_bounds__(kGatherThreads, 6) gather_rows_slot_kernel(
    const int32_t* __restrict__ rowptr, const int32_t* __restrict__ vstart, const int32_t* __restrict__ inc,
    const uint8_t* __restrict__ slot, const double* __restrict__ ev, int nv, double* __restrict__ vals) {
  __shared__ double acc_all[(kGatherThreads / 4) * (kSlotRowMax + 1)];
  const int b = threadIdx.x & 3;
  double* acc = acc_all + (threadIdx.x >> 2) * (kSlotRowMax + 1);
  const int v = blockIdx.x * (kGatherThreads / 4) + (threadIdx.x >> 2);
  int rb = 0, len = 0, q0 = 0, q1 = 0;
  if (v < nv) {
    rb = rowptr[v];
    len = rowptr[v + 1] - rb;
    q0 = vstart[v];
    q1 = vstart[v + 1];
  }
  for (int s = b; s < len; s += 4) acc[s] = 0.0;
  __syncwarp();
  // every row of the warp takes the trips of its longest one, so the warp stays together
  constexpr int U = 4;
  const int trips = (int)__reduce_max_sync(0xffffffffu, (unsigned)(q1 - q0));
  if (b >= K) q1 = q0;  // triangles leave the fourth lane idle
  int sl[U];
  double r[U];
  auto load = [&](int q) {
#pragma unroll
    for (int u = 0; u < U; u++)
      if (q + u < q1) {
        sl[u] = slot[(int64_t)(q + u) * K + b];
        r[u] = ev[(int64_t)inc[q + u] * 4 + b];
      }
  };
  load(q0);
  for (int t = 0; t < trips; t += U) {
    const int q = q0 + t;
    int at[U];
    double w[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      at[u] = sl[u];
      w[u] = r[u];
    }
    load(q + U);
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (REPEATS) {
        for (int turn = 0; turn < K; turn++) {
          if (q + u < q1 && at[u] >> kSlotTurn == turn) acc[at[u] & ((1 << kSlotTurn) - 1)] += w[u];
          __syncwarp();
        }
      } else {
        if (q + u < q1) acc[at[u]] += w[u];
        __syncwarp();  // a column's next contribution may come from another lane of the row
      }
    }
  }
  __syncwarp();
  for (int s = b; s < len; s += 4) vals[rb + s] = acc[s];
}

// One thread per row, rows of any length: contributions of the incident elements, in
// element order, their places found by binary search.
__global__ void gather_rows_kernel(const int32_t* __restrict__ rowptr, const int32_t* __restrict__ cols,
                                   const int32_t* __restrict__ vstart, const int32_t* __restrict__ inc,
                                   const int32_t* __restrict__ conn, const double* __restrict__ ev, int nv,
                                   int k, double* __restrict__ vals, int32_t* bad) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
    int rb = rowptr[v], re = rowptr[v + 1];
    for (int s = rb; s < re; s++) vals[s] = 0.0;
    for (int q = vstart[v]; q < vstart[v + 1]; q++) {
      int code = inc[q];
      int e = code / k;
      for (int b = 0; b < k; b++) {
        int col = conn[(int64_t)e * k + b];
        int s = lower_bound_i32(cols, rb, re, col);
        if (s >= re || cols[s] != col) {
          atomicExch(bad, 1);
          continue;
        }
        vals[s] += ev[(int64_t)code * 4 + b];
      }
    }
  }
}

// Per element: (measure / (k (k + 1)), sum of f over its vertices).  Bound by the FP64 pipe
// (33 operations per tetrahedron).  60^3 cells (1.3 M elements): 90 us (two divisions:
// 113 us).
template <int K>
__global__ void element_load_kernel(const double* __restrict__ xyz, const int32_t* __restrict__ conn,
                                    const double* __restrict__ f, int64_t ne, double2* __restrict__ part) {
  constexpr int k = K;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += (int64_t)gridDim.x * blockDim.x) {
    double meas;
    if (k == 4) {
      double x[4], y[4], z[4];
      for (int a = 0; a < 4; a++) {
        int v = conn[e * 4 + a];
        x[a] = xyz[(int64_t)v * 3];
        y[a] = xyz[(int64_t)v * 3 + 1];
        z[a] = xyz[(int64_t)v * 3 + 2];
      }
      double a1 = x[1] - x[3], a2 = y[1] - y[3], a3 = z[1] - z[3];
      double b1 = x[2] - x[3], b2 = y[2] - y[3], b3 = z[2] - z[3];
      double c1 = x[0] - x[3], c2 = y[0] - y[3], c3 = z[0] - z[3];
      meas = fabs(c1 * (a2 * b3 - a3 * b2) + c2 * (a3 * b1 - a1 * b3) + c3 * (a1 * b2 - a2 * b1));
      meas = div_const<6>(meas);
    } else {
      int v0 = conn[e * 3], v1 = conn[e * 3 + 1], v2 = conn[e * 3 + 2];
      double x0 = xyz[(int64_t)v0 * 3], y0 = xyz[(int64_t)v0 * 3 + 1];
      double x1 = xyz[(int64_t)v1 * 3], y1 = xyz[(int64_t)v1 * 3 + 1];
      double x2 = xyz[(int64_t)v2 * 3], y2 = xyz[(int64_t)v2 * 3 + 1];
      meas = fabs(x0 * y2 - x0 * y1 + x1 * y0 - x1 * y2 + x2 * y1 - x2 * y0) / 2.0;
    }
    double fs = 0;
#pragma unroll
    for (int a = 0; a < k; a++) fs += f[conn[e * k + a]];
    part[e] = make_double2(div_const<K*(K + 1)>(meas), fs);
  }
}

// b_v = sum over the incident elements, in element order (eight in flight).  60^3 cells:
// 39 us (two arrays, one element at a time: 44 us).
template <int K>
__global__ void gather_load_kernel(const int32_t* __restrict__ vstart, const int32_t* __restrict__ inc,
                                   const double2* __restrict__ part, const double* __restrict__ f, int nv,
                                   double* __restrict__ b) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
    double s = 0.0;
    const double fv = f[v];
    const int q1 = vstart[v + 1];
    for (int q0 = vstart[v]; q0 < q1; q0 += 8) {
      double2 p[8];
#pragma unroll
      for (int u = 0; u < 8; u++) p[u] = part[inc[min(q0 + u, q1 - 1)] / K];
#pragma unroll
      for (int u = 0; u < 8; u++)
        if (q0 + u < q1) s += p[u].x * (p[u].y + fv);
    }
    b[v] = s;
  }
}

__global__ void dirichlet_kernel(const int32_t* rowptr, const int32_t* cols, double* vals, const uint8_t* mask, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    bool mi = mask[i] != 0;
    for (int e = rowptr[i]; e < rowptr[i + 1]; e++) {
      int j = cols[e];
      if (mi || mask[j]) vals[e] = (i == j) ? 1.0 : 0.0;
    }
  }
}

// dL/dtheta_e = -c_e * vol_e * grad(lambda)_e . grad(u)_e for P1 tetrahedra: the
// derivative of lambda^T A(theta) u through the stiffness term c_e K_e with
// c_e = exp(theta_e) (the mass term does not depend on theta).
__global__ void grad3d_kernel(const double* __restrict__ xyz, const int32_t* __restrict__ conn,
                              const int32_t* __restrict__ labels, const double* __restrict__ coef, int64_t ne,
                              const double* __restrict__ lam, const double* __restrict__ u,
                              double* __restrict__ grad) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += (int64_t)gridDim.x * blockDim.x) {
    double det, g[4][3];
    tet_gradients(xyz, conn, e, det, g);
    const double vol = fabs(det) / 6.0;
    double gl[3] = {0.0, 0.0, 0.0}, gu[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int a = 0; a < 4; a++) {
      const int v = conn[e * 4 + a];
      const double la = lam[v], ua = u[v];
#pragma unroll
      for (int d = 0; d < 3; d++) {
        gl[d] = fma(la, g[a][d], gl[d]);
        gu[d] = fma(ua, g[a][d], gu[d]);
      }
    }
    const double co = coef ? coef[e] : (labels ? label_coef(labels[e]) : 1.0);
    grad[e] = -co * vol * (gl[0] * gu[0] + gl[1] * gu[1] + gl[2] * gu[2]);
  }
}

// The same for P1 triangles (basis gradients from the 3x3 cofactor inverse).
__global__ void grad2d_kernel(const double* __restrict__ xyz, const int32_t* __restrict__ conn,
                              const double* __restrict__ coef, int64_t ne, const double* __restrict__ lam,
                              const double* __restrict__ u, double* __restrict__ grad) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += (int64_t)gridDim.x * blockDim.x) {
    double x[3], y[3], la[3], ua[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const int v = conn[e * 3 + a];
      x[a] = xyz[(int64_t)v * 3];
      y[a] = xyz[(int64_t)v * 3 + 1];
      la[a] = lam[v];
      ua[a] = u[v];
    }
    const double area = fabs(x[0] * y[2] - x[0] * y[1] + x[1] * y[0] - x[1] * y[2] + x[2] * y[1] - x[2] * y[0]) / 2.0;
    const double det = x[0] * y[1] + x[1] * y[2] + x[2] * y[0] - x[0] * y[2] - x[2] * y[1] - x[1] * y[0];
    // gradient of basis a: ((y[b] - y[c]) / det, (x[c] - x[b]) / det) with (a, b, c) cyclic
    double gl[2] = {0.0, 0.0}, gu[2] = {0.0, 0.0};
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const int b = (a + 1) % 3, c = (a + 2) % 3;
      const double gx = (y[b] - y[c]) / det, gy = (x[c] - x[b]) / det;
      gl[0] = fma(la[a], gx, gl[0]);
      gl[1] = fma(la[a], gy, gl[1]);
      gu[0] = fma(ua[a], gx, gu[0]);
      gu[1] = fma(ua[a], gy, gu[1]);
    }
    const double co = coef ? coef[e] : 1.0;
    grad[e] = -co * area * (gl[0] * gu[0] + gl[1] * gu[1]);
  }
}

__global__ void mask_rows_kernel(int n, const uint8_t* __restrict__ mask, const double* __restrict__ in,
                                 double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (mask && mask[i]) ? 0.0 : in[i];
}

__global__ void row_length_kernel(const int32_t* rowptr, int n, int32_t* len) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) len[i] = rowptr[i + 1] - rowptr[i];
}

// Longest row of the level-0 pattern.
int reduce_max_row_length(Ctx& c) {
  DBuf<int32_t> len(c.A.n > 0 ? c.A.n : 1, c.stream);
  FG_LAUNCH(row_length_kernel, grid_for(c.A.n, 256), 256, 0, c.stream, c.A.rp.p, c.A.n, len.p);
  return reduce_max(len.p, c.A.n, c.stream);
}

// The element matrices into the element table (4 doubles per incidence).
void element_matrices(Ctx& c, const double* coef, double lambda, double* ev) {
  cudaStream_t s = c.stream;
  Mesh& M = c.mesh;
  const int g = grid_for(M.ne, 128);
  const int32_t* lab = M.has_labels ? M.labels.p : nullptr;
  if (M.k == 4) {
    auto k = lambda != 0.0 ? element3d_kernel<true> : element3d_kernel<false>;
    FG_LAUNCH(k, g, 128, 0, s, M.xyz.p, M.conn.p, lab, coef, M.ne, lambda, ev);
  } else {
    auto k = lambda != 0.0 ? element2d_kernel<true> : element2d_kernel<false>;
    FG_LAUNCH(k, g, 128, 0, s, M.xyz.p, M.conn.p, coef, M.ne, lambda, ev);
  }
}

// Row gather of the element table into the operator's values (slot map when built).
void gather_rows(Ctx& c, const double* ev, double* vals) {
  cudaStream_t s = c.stream;
  Mesh& M = c.mesh;
  if (M.slot.n) {
    auto k = M.repeats ? (M.k == 4 ? gather_rows_slot_kernel<4, true> : gather_rows_slot_kernel<3, true>)
                       : (M.k == 4 ? gather_rows_slot_kernel<4, false> : gather_rows_slot_kernel<3, false>);
    FG_LAUNCH(k, grid_for(M.nv, kGatherThreads / 4), kGatherThreads, 0, s, c.A.rp.p, M.vstart.p, M.inc.p, M.slot.p, ev,
              (int)M.nv, vals);
    return;
  }
  DBuf<int32_t> bad(1, s);
  bad.zero();
  FG_LAUNCH(gather_rows_kernel, grid_for(M.nv, 128), 128, 0, s, c.A.rp.p, c.A.ci.p, M.vstart.p, M.inc.p, M.conn.p,
            ev, (int)M.nv, M.k, vals, bad.p);
  FG_REQUIRE(read_scalar(bad.p, s) == 0, FEMGPU_ERR_INVALID, "element entry outside the pattern");
}

}  // namespace

void build_mesh_pattern(Ctx& c) {
  cudaStream_t s = c.stream;
  Mesh& M = c.mesh;
  const int nv = (int)M.nv, k = M.k;
  const int64_t nslots = M.ne * k;
  c.mesh_pattern = c.mesh_graph = false;
  DBuf<int32_t> deg(nv + 1, s), bad(1, s);
  deg.zero();
  bad.zero();
  FG_LAUNCH(incidence_count_kernel, grid_for(nslots, 256), 256, 0, s, M.conn.p, nslots, deg.p, nv, bad.p);
  FG_REQUIRE(read_scalar(bad.p, s) == 0, FEMGPU_ERR_INVALID, "element connectivity references a vertex out of range");
  M.vstart.alloc(nv + 1, s);
  int64_t total = exclusive_scan(deg.p, M.vstart.p, nv, s);
  FG_REQUIRE(total == nslots, FEMGPU_ERR_INVALID, "incidence count mismatch");
  M.inc.alloc(nslots, s);
  DBuf<int32_t> cursor(nv, s);
  cursor.zero();
  FG_LAUNCH(incidence_fill_kernel, grid_for(nslots, 256), 256, 0, s, M.conn.p, nslots, M.vstart.p, cursor.p, M.inc.p);
  segmented_sort_i32(M.inc.p, M.vstart.p, nv, nullptr, s);
  // candidate columns: all vertices of every incident element (includes the row itself)
  DBuf<int32_t> ccount(nv + 1, s), coff(nv + 1, s);
  FG_LAUNCH(times_k_kernel, grid_for(nv, 256), 256, 0, s, deg.p, nv, k, ccount.p);
  int64_t ncand = exclusive_scan(ccount.p, coff.p, nv, s);
  FG_REQUIRE(ncand < INT32_MAX, FEMGPU_ERR_LIMIT, "pattern candidate count exceeds int32");
  DBuf<int32_t> cand(ncand > 0 ? ncand : 1, s);
  FG_LAUNCH(candidates_kernel, grid_for(nv, 128), 128, 0, s, M.conn.p, M.vstart.p, M.inc.p, coff.p, nv, k, cand.p);
  DBuf<int32_t> ucount(nv + 1, s);
  segmented_sort_i32(cand.p, coff.p, nv, ucount.p, s);
  // isolated vertices still get their diagonal
  c.A.n = c.A.m = nv;
  c.A.rp.alloc(nv + 1, s);
  int64_t nnz = exclusive_scan(ucount.p, c.A.rp.p, nv, s);
  c.A.nnz = nnz;
  c.A.ci.alloc(nnz, s);
  c.A.v.alloc(nnz, s);
  c.A.v.zero();
  FG_LAUNCH(compact_rows_kernel, grid_for((int64_t)nv * 32, 256), 256, 0, s, cand.p, coff.p, c.A.rp.p, nv, c.A.ci.p);
  // slot map for the assembly's row gather, when every row fits its shared-memory sums
  M.slot.release();
  c.A_max_row = reduce_max_row_length(c);
  if (c.A_max_row <= kSlotRowMax) {
    M.slot.alloc((size_t)nslots * k, s);
    DBuf<int32_t> found(2, s);
    found.zero();
    FG_LAUNCH(slot_map_kernel, grid_for(nv, 128), 128, 0, s, c.A.rp.p, c.A.ci.p, M.vstart.p, M.inc.p, M.conn.p, nv,
              k, M.slot.p, found.p, found.p + 1);
    int32_t h[2];
    found.download(h, 2);
    FG_CUDA(cudaStreamSynchronize(s));
    FG_REQUIRE(h[0] == 0, FEMGPU_ERR_INVALID, "element vertex outside the pattern");
    M.repeats = h[1] != 0;
  }
  // level-0 aggregation graph: the pattern without self loops
  c.gxadj.alloc(nv + 1, s);
  c.gadj.alloc(nnz - nv > 0 ? nnz - nv : 1, s);
  FG_LAUNCH(graph_from_pattern_kernel, grid_for(nv, 256), 256, 0, s, c.A.rp.p, c.A.ci.p, nv, c.gxadj.p, c.gadj.p);
  c.graph_nnz = nnz - nv;
  c.mesh_pattern = c.mesh_graph = true;
}

void assemble_operator(Ctx& c, const double* coef_host, double lambda, bool coef_on_device) {
  cudaStream_t s = c.stream;
  Mesh& M = c.mesh;
  const int64_t ne = M.ne;
  const int k = M.k;
  if (!c.mesh_pattern) {  // a matrix was set since the mesh
    c.has_matrix = false;
    build_mesh_pattern(c);
  }
  if (k == 4) {
    double t[10];
    tet_mass_table(t);
    FG_CUDA(cudaMemcpyToSymbolAsync(c_tet_mass, t, sizeof(t), 0, cudaMemcpyHostToDevice, s));
  } else {
    double zx[6], wx[6], zy[6], wy[6], q[36];
    tri_quadrature_table(zx, wx, zy, wy);
    for (int i = 0; i < 6; i++) {
      q[i] = wx[i];
      q[6 + i] = wy[i];
      q[12 + i] = 1 - zx[i];
      q[18 + i] = 1 + zx[i];
      q[24 + i] = 1 - zy[i];
      q[30 + i] = 1 + zy[i];
    }
    FG_CUDA(cudaMemcpyToSymbolAsync(c_tri_q, q, sizeof(q), 0, cudaMemcpyHostToDevice, s));
  }
  DBuf<double>& coef = c.coef;  // kept for the adjoint gradient
  c.lambda_mass = lambda;
  coef.release();
  if (coef_host) {
    coef.alloc(ne, s);
    if (coef_on_device)
      FG_CUDA(cudaMemcpyAsync(coef.p, coef_host, ne * sizeof(double), cudaMemcpyDeviceToDevice, s));
    else
      coef.upload(coef_host, ne);
  }
  DBuf<double> ev((size_t)ne * k * 4, s);
  element_matrices(c, coef.p, lambda, ev.p);
  gather_rows(c, ev.p, c.A.v.p);
}

void load_vector(Ctx& c, const double* f_host, double* b_host) {
  cudaStream_t s = c.stream;
  Mesh& M = c.mesh;
  DBuf<double> f(M.nv, s), b(M.nv, s);
  DBuf<double2> part(M.ne, s);
  f.upload(f_host, M.nv);
  load_vector_enqueue(c, f.p, b.p, part.p);
  b.download(b_host, M.nv);
  FG_CUDA(cudaStreamSynchronize(s));
}

void load_vector_enqueue(Ctx& c, const double* d_f, double* d_b, double2* part) {
  cudaStream_t s = c.stream;
  Mesh& M = c.mesh;
  auto el = M.k == 4 ? element_load_kernel<4> : element_load_kernel<3>;
  auto ga = M.k == 4 ? gather_load_kernel<4> : gather_load_kernel<3>;
  FG_LAUNCH(el, grid_for(M.ne, 256), 256, 0, s, M.xyz.p, M.conn.p, d_f, M.ne, part);
  FG_LAUNCH(ga, grid_for(M.nv, 128), 128, 0, s, M.vstart.p, M.inc.p, part, d_f, (int)M.nv, d_b);
}

void zero_dirichlet_rows(Ctx& c, const double* d_in, double* d_out) {
  const int n = c.A.n;
  FG_LAUNCH(mask_rows_kernel, grid_for(n, 256), 256, 0, c.stream, n, c.dmask.n ? c.dmask.p : nullptr, d_in, d_out);
}

void element_log_coef_gradient(Ctx& c, const double* d_lam, const double* d_u, double* d_grad) {
  Mesh& M = c.mesh;
  const double* coef = c.coef.n ? c.coef.p : nullptr;
  if (M.k == 4)
    FG_LAUNCH(grad3d_kernel, grid_for(M.ne, 128), 128, 0, c.stream, M.xyz.p, M.conn.p,
              M.has_labels ? M.labels.p : nullptr, coef, M.ne, d_lam, d_u, d_grad);
  else
    FG_LAUNCH(grad2d_kernel, grid_for(M.ne, 128), 128, 0, c.stream, M.xyz.p, M.conn.p, coef, M.ne, d_lam, d_u,
              d_grad);
}

void profile_assembly(Ctx& c, int which, int reps, double* ms, double* bytes) {
  FG_REQUIRE(c.has_mesh && c.assembled_from_mesh, FEMGPU_ERR_NOT_READY, "no operator assembled from the mesh");
  cudaStream_t s = c.stream;
  Mesh& M = c.mesh;
  const int64_t ne = M.ne, nv = M.nv, nnz = c.A.nnz;
  const int k = M.k;
  DBuf<double> ev((size_t)ne * k * 4, s), vals(nnz, s);
  const double* coef = c.coef.n ? c.coef.p : nullptr;
  auto element = [&]() { element_matrices(c, coef, c.lambda_mass, ev.p); };
  auto gather = [&]() { gather_rows(c, ev.p, vals.p); };
  element();
  auto run = [&]() {
    if (which == 6) element();
    else gather();
  };
  if (which == 6)  // connectivity, coefficient and entries per element, coordinates once per vertex
    *bytes = (double)ne * (4.0 * k + (coef ? 8.0 : 0.0) + 32.0 * k) + 24.0 * nv;
  else if (M.slot.n)  // row and incidence offsets, incidence lists, slot map, element entries, values out
    *bytes = 8.0 * (nv + 1) + 4.0 * k * ne + 1.0 * k * k * ne + 32.0 * k * ne + 8.0 * nnz;
  else  // row offsets, columns, incidence offsets and lists, the incident elements' vertices and entries, values out
    *bytes = 8.0 * (nv + 1) + 4.0 * nnz + 4.0 * k * ne + 4.0 * k * ne + 32.0 * k * ne + 8.0 * nnz;
  for (int i = 0; i < 3; i++) run();
  cudaEvent_t e0, e1;
  FG_CUDA(cudaEventCreate(&e0));
  FG_CUDA(cudaEventCreate(&e1));
  FG_CUDA(cudaEventRecord(e0, s));
  for (int i = 0; i < reps; i++) run();
  FG_CUDA(cudaEventRecord(e1, s));
  FG_CUDA(cudaEventSynchronize(e1));
  float t = 0;
  FG_CUDA(cudaEventElapsedTime(&t, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  *ms = t / reps;
}

void apply_dirichlet(Ctx& c, const uint8_t* mask_host) {
  cudaStream_t s = c.stream;
  DBuf<uint8_t>& mask = c.dmask;  // kept for the adjoint right-hand side
  mask.alloc(c.A.n, s);
  mask.upload(mask_host, c.A.n);
  FG_LAUNCH(dirichlet_kernel, grid_for(c.A.n, 256), 256, 0, s, c.A.rp.p, c.A.ci.p, c.A.v.p, mask.p, c.A.n);
  FG_CUDA(cudaStreamSynchronize(s));
}

}  // namespace femgpu
