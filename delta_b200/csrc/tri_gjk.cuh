// tri_gjk.cuh -- GJK distance between two triangles with Johnson's sub-simplex
// projection, the arithmetic of gjk.cpp:302-460 (Solfec's gjk) for na = nb = 3.
#pragma once
#include "real.cuh"

namespace delta {

// Simplex vertex: Minkowski point w = A[ia] - B[ib], id = ia | ib << 2.
template <class R>
struct GjkVertex {
  R w[3];
  int id;
};

// project(), gjk.cpp:302-414, for a simplex of n = 1..4 points.  Subsets are tried in the
// order of gjk.cpp:120-135 (the order decides which sub-simplex is accepted first; those
// of n points are the first 2^n - 1).  All of them are evaluated, whatever n is, and the
// first acceptable one is selected: every index is a compile-time constant, so the
// simplex, the dot products and the cofactors stay in registers (indexed at run time they
// lived in local memory), and the lanes of a warp run the same instructions whatever
// simplex each holds and whichever subset it accepts.
template <class R>
__device__ __forceinline__ int gjk_project(GjkVertex<R> *w, int n, R *l, R *v) {
  constexpr int N = 4;
  constexpr int subsets[15] = {1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 12, 11, 13, 14, 15};
  R dots[N][N], dl[1 << N][N];
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = i; j < N; ++j) {
      dots[i][j] = dot3(w[i].w, w[j].w);
      dots[j][i] = dots[i][j];
    }
  int sub = 0;  // the first acceptable subset (0: none yet)
  R ls[N];
#pragma unroll
  for (int i = 0; i < N; ++i) ls[i] = R(0.0);
#pragma unroll
  for (int m = 0; m < (1 << N) - 1; ++m) {
    const int s = subsets[m];
    bool ok = s < (1 << n);
    int k = -1;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (s & (1 << i)) {
        const int o = s & ~(1 << i);
        if (k < 0) k = i;
        if (o == 0) {
          dl[s][i] = R(1.0);
        } else {
          dl[s][i] = dl[o][i];
          if (dl[s][i] <= R(0.0)) ok = false;
        }
      }
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (!(s & (1 << j))) {
        if ((s & (s - 1)) == 0) {
          dl[s][j] = dots[k][k] - dots[k][j];
        } else {
          dl[s][j] = R(0.0);
#pragma unroll
          for (int i = 0; i < N; ++i)
            if (s & (1 << i)) dl[s][j] += dl[s][i] * (dots[i][k] - dots[i][j]);
        }
        if (dl[s][j] > R(0.0) && j < n) ok = false;
      }
    ok = ok && sub == 0;
    sub = ok ? s : sub;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (s & (1 << i)) ls[i] = ok ? dl[s][i] : ls[i];
  }
  if (sub == 0) return 0;
  // keep the subset's points, in order: drop the others from the last to the first
#pragma unroll
  for (int i = N - 1; i >= 0; --i)
    if (!(sub & (1 << i))) {
#pragma unroll
      for (int j = i; j + 1 < N; ++j) {
        w[j] = w[j + 1];
        ls[j] = ls[j + 1];
      }
    }
  const int o = __popc(sub);
  R sum = R(0.0);
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (i < o) sum += ls[i];
  R u[3] = {R(0.0), R(0.0), R(0.0)};
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (i < o) {
      l[i] = ls[i] / sum;
#pragma unroll
      for (int k = 0; k < 3; ++k) u[k] = u[k] + l[i] * w[i].w[k];
    }
#pragma unroll
  for (int k = 0; k < 3; ++k) v[k] = n == 1 ? w[0].w[k] : u[k];  // a point is its own projection
  return o;
}

__device__ __forceinline__ bool same_bits(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
__device__ __forceinline__ bool same_bits(xf64 a, xf64 b) {
  return __double_as_longlong(a.v) == __double_as_longlong(b.v);
}

// gjk(a,3,b,3,p,q), gjk.cpp:418-460; GEOMETRIC_EPSILON = 1e-6 (gjk.cpp:102): start(), then
// step() while it returns true, then points().  The support points are the first extreme
// vertex (gjk.cpp:141-165).
//
// Rounding often keeps the error bound above the tolerance, and the reference then
// repeats a short cycle of simplices until its 36th iteration.  An iteration is a function
// of (the simplex' points in order, v, mi) alone, so when that state equals, bit for bit,
// the state saved lam iterations ago, whole cycles are left out: the state after the 36th
// iteration is that after (36 - j) mod lam more.  The state is compared with the last one
// (in FP32 60% of the microbenchmark's pairs end in a fixed point, most by the 7th
// iteration) and with one saved at iterations 1, 2, 4, 8, 16 (Brent's method).
template <class R>
struct Gjk {
  static constexpr int kMax = 36;
  GjkVertex<R> w[4];
  R v[3], l[4], mi, vlen;
  R sv[3], smi;  // the saved state, its simplex and iteration
  int skey, sj, key;
  int n, j;
  bool cut;  // whole cycles already left out

  __device__ __forceinline__ bool start(const R A[3][3], const R B[3][3]) {
    mi = R(0.0);
    n = j = sj = 0;
    skey = key = -1;
    cut = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      w[k].w[0] = w[k].w[1] = w[k].w[2] = l[k] = R(0.0);
      w[k].id = 0;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) sv[k] = v[k] = A[0][k] - B[0][k];
    smi = mi;
    vlen = sqrt_(dot3(v, v));
    return vlen > R(1E-6);
  }

  // one iteration; false when it was the last
  __device__ __forceinline__ bool step(const R A[3][3], const R B[3][3]) {
    const R GEPS = R(1E-6);
    ++j;
    int ia = 0, ib = 0;
    R best = R(1.7976931348623157e308);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const R dd = dot3(A[q], v);
      if (dd < best) { best = dd; ia = q; }
    }
    best = R(-1.7976931348623157e308);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const R dd = dot3(B[q], v);
      if (dd > best) { best = dd; ib = q; }
    }
    GjkVertex<R> nw;
    nw.id = ia | (ib << 2);
#pragma unroll
    for (int k = 0; k < 3; ++k)
      nw.w[k] = (ia == 0 ? A[0][k] : (ia == 1 ? A[1][k] : A[2][k])) - (ib == 0 ? B[0][k] : (ib == 1 ? B[1][k] : B[2][k]));
    const R dlt = dot3(v, nw.w) / vlen;
    const R lmi = mi, lv[3] = {v[0], v[1], v[2]};
    const int lkey = key;
    mi = (mi > dlt) ? mi : dlt;
    if (!((vlen - mi) > GEPS)) return false;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k == n) w[k] = nw;
    n = gjk_project(w, n + 1, l, v);
    vlen = sqrt_(dot3(v, v));
    // the simplex in order: count, and 4 bits a point
    key = n | (n > 0 ? w[0].id << 3 : 0) | (n > 1 ? w[1].id << 7 : 0) | (n > 2 ? w[2].id << 11 : 0) |
          (n > 3 ? w[3].id << 15 : 0);
    if (repeats(lkey, lmi, lv)) return false;
    if (!cut && repeats(skey, smi, sv)) {
      j = kMax - (kMax - j) % (j - sj);
      cut = true;
    } else if ((j & (j - 1)) == 0) {
      skey = key;
      sj = j;
      smi = mi;
      sv[0] = v[0];
      sv[1] = v[1];
      sv[2] = v[2];
    }
    return vlen > GEPS && n < 4 && j < kMax;
  }

  __device__ __forceinline__ bool repeats(int k, R m, const R *u) const {
    return key == k && same_bits(mi, m) && same_bits(v[0], u[0]) && same_bits(v[1], u[1]) && same_bits(v[2], u[2]);
  }

  __device__ __forceinline__ void points(const R A[3][3], const R B[3][3], R pq[6]) const {
    if (n == 0) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        pq[k] = A[0][k];
        pq[3 + k] = B[0][k];
      }
      return;
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) pq[k] = R(0.0);
#pragma unroll
    for (int m = 3; m >= 0; --m)
      if (m < n) {
        const int ia = w[m].id & 3, ib = w[m].id >> 2;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const R av = ia == 0 ? A[0][k] : (ia == 1 ? A[1][k] : A[2][k]);
          const R bv = ib == 0 ? B[0][k] : (ib == 1 ? B[1][k] : B[2][k]);
          pq[k] = pq[k] + l[m] * av;
          pq[3 + k] = pq[3 + k] + l[m] * bv;
        }
      }
  }
};

template <class R>
__device__ __forceinline__ void gjk_ref(const R A[3][3], const R B[3][3], R pq[6]) {
  Gjk<R> g;
  for (bool more = g.start(A, B); more;) more = g.step(A, B);
  g.points(A, B, pq);
}

}  // namespace delta
