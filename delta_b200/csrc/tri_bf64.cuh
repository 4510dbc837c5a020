// tri_bf64.cuh -- the FP64 bfSolver (reference arithmetic) on triangles in shared memory.
#pragma once
#include "tri_ref.cuh"

namespace delta {

// FP64 bfSolver (bf.cpp:217-1178): the 15 evaluations, comparisons and results of
// bf_solve_lean.  The kernels keep the triangles in shared memory (plane, pair) and load a
// feature's vertices from there, at a row that is the same for the whole warp, in a column
// of the lane's own: nothing of a pair but the running minimum stays in registers between
// features (the register copies rotated by bf_solve_lean held 36 doubles).
struct BfBest {
  xf64 d, p0, p1;  // distance and the winner's parameters
  int id;          // edge pair 3 ea + eb; vertex-face 3 face + vertex (face 0: A's)
  __device__ __forceinline__ void start() {
    d = xf64(1E+30);
    p0 = p1 = xf64(0.0);
    id = 0;
  }
  __device__ __forceinline__ void take(xf64 dist, xf64 x0, xf64 x1, int j) {
    if (dist < d) {
      d = dist;
      p0 = x0;
      p1 = x1;
      id = j;
    }
  }
};

template <int COLS>
struct BfTile {
  double v[18][COLS];
  __device__ __forceinline__ void vertex(int t, int col, xf64 x[3]) const {  // A's 0..2, B's 3..5
#pragma unroll
    for (int k = 0; k < 3; ++k) x[k] = xf64(v[3 * t + k][col]);
  }
  // the edge pairs of A's edge ea, in order
  __device__ __forceinline__ void edges(int ea, int col, BfBest &best) const {
    xf64 HA[3], TA[3];
    vertex(ea, col, HA);
    vertex(ea == 2 ? 0 : ea + 1, col, TA);
#pragma unroll 1
    for (int eb = 0; eb < 3; ++eb) {
      xf64 HB[3], TB[3], sc, tc;
      vertex(3 + eb, col, HB);
      vertex(eb == 2 ? 3 : 4 + eb, col, TB);
      const xf64 d = seg_seg_ref(HA, TA, HB, TB, sc, tc);
      best.take(d, sc, tc, 3 * ea + eb);
    }
  }
  // the vertices of the other triangle against face 0 (A) or 1 (B), in order
  __device__ __forceinline__ void faces(int face, int col, BfBest &best) const {
    xf64 T0[3], T1[3], T2[3];
    vertex(3 * face, col, T0);
    vertex(3 * face + 1, col, T1);
    vertex(3 * face + 2, col, T2);
#pragma unroll 1
    for (int j = 0; j < 3; ++j) {
      xf64 X[3], s, t;
      vertex(3 * (1 - face) + j, col, X);
      const xf64 d = pt_tri_ref(T0, T1, T2, X, s, t);
      best.take(d, s, t, 3 * face + j);
    }
  }
  // the winner's points (seg_seg_points, pt_tri_points): e the edge pairs' best, f the faces'
  __device__ __forceinline__ void points(int col, const BfBest &e, const BfBest &f, xf64 pq[6]) const {
    if (f.d > e.d) {
      const int ea = e.id / 3, eb = e.id % 3;
      xf64 HA[3], TA[3], HB[3], TB[3];
      vertex(ea, col, HA);
      vertex(ea == 2 ? 0 : ea + 1, col, TA);
      vertex(3 + eb, col, HB);
      vertex(eb == 2 ? 3 : 4 + eb, col, TB);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        pq[k] = TA[k] + ((HA[k] - TA[k]) * e.p0);
        pq[3 + k] = TB[k] + ((HB[k] - TB[k]) * e.p1);
      }
    } else {
      const bool onA = f.id < 3;
      xf64 T0[3], T1[3], T2[3], X[3];
      vertex(onA ? 0 : 3, col, T0);
      vertex(onA ? 1 : 4, col, T1);
      vertex(onA ? 2 : 5, col, T2);
      vertex(onA ? 3 + f.id : f.id - 3, col, X);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const xf64 face = T0[k] + ((T2[k] - T0[k]) * f.p1) + ((T1[k] - T0[k]) * f.p0);
        pq[k] = onA ? face : X[k];
        pq[3 + k] = onA ? X[k] : face;
      }
    }
  }
  // a whole pair in one thread
  __device__ __forceinline__ void solve(int col, xf64 pq[6]) const {
    BfBest e, f;
    e.start();
    f.start();
#pragma unroll 1
    for (int ea = 0; ea < 3; ++ea) edges(ea, col, e);
#pragma unroll 1
    for (int face = 0; face < 2; ++face) faces(face, col, f);
    points(col, e, f, pq);
  }
};

}  // namespace delta
