// The staging shared by the point-parallel Gauss-point kernels (general.cu's exact form,
// general_fast.cu's fast form): a block of 256 threads takes 32 consecutive elements, warp g their
// Gauss point g, lane l element l. So every array indexed by element ([k * P + e]) is read and
// written as whole lines, the point's constants are the same for a warp, and the points' values meet
// in shared memory, each warp's row of 32 doubles free of bank conflicts.
//
// What bounds these kernels is latency at 16 warps per SM (128 registers), the FP64 pipe at 46 % of
// its rate (about 5,200 operations per element without the mass term). A thread per element (before)
// held 255 registers, 8 warps per SM, and its eight points ran one after the other. Measured, B200:
// caches warm: the exact operator with mass on 49,321 distorted bricks 51.1 -> 36.8 us, on 5,120 J2
// bricks 17.5 -> 7.1 us, on 15,700 J2 bricks 17.5 -> 11.9 us; the damped fast force on 64,000 bricks
// 46.1 -> 46.9 us (the undamped one 39 us with the gather; general_fast.cu). A thread per element stays
// where it is faster: points_apply_pays in general.cu.
#pragma once

#include "force.hpp"

namespace fx {
namespace points {

constexpr int kEl = 32;               // elements per block
constexpr int kThreads = 8 * kEl;     // a thread per Gauss point
constexpr int kEdges = 36;            // 12 edge vectors of 3 components

// The edges whose components the Jacobian's columns sum (column = edge / 4, in the order of
// brick_gp.cuh's sums): from corner kFrom to corner kTo.
__device__ constexpr int8_t kTo[12] = {1, 2, 5, 6, 2, 3, 6, 7, 4, 5, 6, 7};
__device__ constexpr int8_t kFrom[12] = {0, 3, 4, 7, 1, 0, 5, 4, 0, 1, 2, 3};

// A Gauss point's shape factors: a, b, c of the four faces (brick_gp.cuh's shape_at, in its order
// (-,-), (+,+), (-,+), (+,-)), and the eight values N.
struct PointTable {
  double a[4], b[4], c[4], N[8];
};
__device__ __forceinline__ void point_table(int gp, PointTable& t) {
  double g[3];
  gauss_point(gp, g);
  const double p1 = 1.0 + g[0], m1 = 1.0 - g[0];
  const double p2 = 1.0 + g[1], m2 = 1.0 - g[1];
  const double p3 = 1.0 + g[2], m3 = 1.0 - g[2];
  t.a[0] = 0.125 * m1 * m2, t.b[0] = 0.125 * m2 * m3, t.c[0] = 0.125 * m1 * m3;
  t.a[1] = 0.125 * p1 * p2, t.b[1] = 0.125 * p2 * p3, t.c[1] = 0.125 * p1 * p3;
  t.a[2] = 0.125 * m1 * p2, t.b[2] = 0.125 * m2 * p3, t.c[2] = 0.125 * m1 * p3;
  t.a[3] = 0.125 * p1 * m2, t.b[3] = 0.125 * p2 * m3, t.c[3] = 0.125 * p1 * m3;
  t.N[0] = t.a[0] * m3, t.N[4] = t.a[0] * p3;
  t.N[2] = t.a[1] * m3, t.N[6] = t.a[1] * p3;
  t.N[3] = t.a[2] * m3, t.N[7] = t.a[2] * p3;
  t.N[1] = t.a[3] * m3, t.N[5] = t.a[3] * p3;
}

// NX staged vectors (the operator's x; the force's u and v), NP partial sums per point and value.
template <int NX, int NP>
struct Stage {
  double edge[kEdges][kEl];
  double x[NX][24][kEl];
  double part[8][NP][24][kEl];
  PointTable tab[8];
  // corner coordinates on their way to the edges (row 3 a + d)
  __device__ double (*corners())[kEl] { return part[0][0]; }
};
// The same for kernels that sum nothing over the points.
template <int NX>
struct Stage<NX, 0> {
  double edge[kEdges][kEl];
  double x[NX][24][kEl];
  double xl[24][kEl];
  PointTable tab[8];
  __device__ double (*corners())[kEl] { return xl; }
};

// The block's elements: their edge vectors and their values of x0 (and x1), by all threads; the point
// tables by eight of them. Elements past `count` stage zeros: a degenerate element, whose points give
// NaN where a kernel evaluates them (it writes nothing of theirs).
template <int NX, int NP>
__device__ __forceinline__ void stage_elements(Stage<NX, NP>& S, const double* __restrict__ coords,
                                               const int32_t* __restrict__ node, const int32_t* __restrict__ eq,
                                               int32_t N, int32_t P, int32_t count, const double* __restrict__ x0,
                                               const double* __restrict__ x1) {
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int32_t e = static_cast<int32_t>(blockIdx.x) * kEl + l;
  const bool ok = e < count;
  int32_t q[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) q[k] = ok ? eq[static_cast<int64_t>(w + 8 * k) * P + e] : -1;
  double(*xl)[kEl] = S.corners();
  const int32_t n = ok ? node[static_cast<int64_t>(w) * P + e] : 0;
#pragma unroll
  for (int d = 0; d < 3; ++d) xl[3 * w + d][l] = ok ? coords[static_cast<int64_t>(d) * N + n] : 0.0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    S.x[0][w + 8 * k][l] = q[k] >= 0 ? x0[q[k]] : 0.0;
    if constexpr (NX == 2)
      if (x1) S.x[1][w + 8 * k][l] = q[k] >= 0 ? x1[q[k]] : 0.0;
  }
  if (l == 0) point_table(w, S.tab[w]);
  __syncthreads();
  for (int k = w; k < 12; k += 8)
#pragma unroll
    for (int d = 0; d < 3; ++d) S.edge[3 * k + d][l] = xl[3 * kTo[k] + d][l] - xl[3 * kFrom[k] + d][l];
  __syncthreads();
}

// The global derivatives and the volume of this thread's point: shape_at's sums in its order, the
// products of a face's factor shared by the two corners that take it with opposite signs.
template <class S>
__device__ __forceinline__ void shape(const S& st, const PointTable& t, int l, double dN[3][8], double& dvol) {
  double J[3][3], A[3][3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    J[d][0] = st.edge[d][l] * t.b[0] + st.edge[3 + d][l] * t.b[3] + st.edge[6 + d][l] * t.b[2] +
              st.edge[9 + d][l] * t.b[1];
    J[d][1] = st.edge[12 + d][l] * t.c[3] + st.edge[15 + d][l] * t.c[0] + st.edge[18 + d][l] * t.c[1] +
              st.edge[21 + d][l] * t.c[2];
    J[d][2] = st.edge[24 + d][l] * t.a[0] + st.edge[27 + d][l] * t.a[3] + st.edge[30 + d][l] * t.a[1] +
              st.edge[33 + d][l] * t.a[2];
  }
  A[0][0] = J[1][1] * J[2][2] - J[1][2] * J[2][1];
  A[0][1] = J[2][1] * J[0][2] - J[2][2] * J[0][1];
  A[0][2] = J[0][1] * J[1][2] - J[0][2] * J[1][1];
  A[1][0] = J[1][2] * J[2][0] - J[1][0] * J[2][2];
  A[1][1] = J[2][2] * J[0][0] - J[2][0] * J[0][2];
  A[1][2] = J[0][2] * J[1][0] - J[0][0] * J[1][2];
  A[2][0] = J[1][0] * J[2][1] - J[1][1] * J[2][0];
  A[2][1] = J[2][0] * J[0][1] - J[2][1] * J[0][0];
  A[2][2] = J[0][0] * J[1][1] - J[0][1] * J[1][0];
  const double det = J[0][0] * A[0][0] + J[0][1] * A[1][0] + J[0][2] * A[2][0];
  const double rdet = 1.0 / det;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double i0 = A[0][c] * rdet, i1 = A[1][c] * rdet, i2 = A[2][c] * rdet;
    double B[4], C[4], D[4];
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      B[f] = t.b[f] * i0;
      C[f] = t.c[f] * i1;
      D[f] = t.a[f] * i2;
    }
    dN[c][0] = -B[0] - C[0] - D[0];
    dN[c][1] = B[0] - C[3] - D[3];
    dN[c][2] = B[3] + C[3] - D[1];
    dN[c][3] = -B[3] + C[0] - D[2];
    dN[c][4] = -B[2] - C[2] + D[0];
    dN[c][5] = B[2] - C[1] + D[3];
    dN[c][6] = B[1] + C[1] + D[1];
    dN[c][7] = -B[1] + C[2] + D[2];
  }
  dvol = det;
}

// epsilon = B u of element l's values u (strain_of's sums in its order)
__device__ __forceinline__ void strain(const double dN[3][8], const double (*u)[kEl], int l, double e[6]) {
#pragma unroll
  for (int c = 0; c < 6; ++c) e[c] = 0.0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const double dx = dN[0][j], dy = dN[1][j], dz = dN[2][j];
    const double u0 = u[3 * j][l], u1 = u[3 * j + 1][l], u2 = u[3 * j + 2][l];
    e[0] += dx * u0;
    e[1] += dy * u1;
    e[2] += dz * u2;
    e[3] += dy * u0 + dx * u1;
    e[4] += dz * u1 + dy * u2;
    e[5] += dz * u0 + dx * u2;
  }
}

// B_j^T s of s = sigma dvol (node_force's sums)
__device__ __forceinline__ void corner_force(const double dN[3][8], const double s[6], int j, double r[3]) {
  const double dx = dN[0][j], dy = dN[1][j], dz = dN[2][j];
  r[0] = dx * s[0] + dy * s[3] + dz * s[5];
  r[1] = dy * s[1] + dx * s[3] + dz * s[4];
  r[2] = dz * s[2] + dy * s[4] + dx * s[5];
}

}  // namespace points
}  // namespace fx
