"""The band of the certified FP32 lower bounds (delta_b200/csrc/tri_cert.cuh) on the CPU.

A feature is left out when its bound, less the band 64 u32 L, exceeds a distance found in FP64
(u32 = 2^-24, L the extent of the pair). Two things are shown here.

The band has room. Derivation, in units of u32 L: the coordinates' rounding moves a point pair
by 2 a component; the difference vector's two multiply-adds and three differences add at most
7; over three components 9 * 1.74 = 16. The squared length, rsqrt (2 ulp) and their product:
8 on the distance, which is at most 1.74 L. The gradient terms r.u / |r| and r.v / |r|: at most
4 roundings of a product of 1.74 each, twice: 14; their product with 1 / |r| and the sum: 4.
Together 42 of the 64. So taking L itself in FP32, which moves it by at most 3 u32 relative,
moves the band by 2e-5 units. The functions of the source are compiled for the host (rsqrt at
both ends of its error) and their error is measured against long double.

The comparison in FP32 decides as in FP64: a float exceeds a double exactly when it exceeds
the double rounded down to a float.
"""
import re
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "delta_b200" / "csrc"

HARNESS = r"""
#include <math.h>
#include <cmath>
#include <cstdlib>
#include <cstdint>
#include <cstdio>
#include <random>
#define __device__
#define __forceinline__ inline
static float g_rsqrt = 1.f;
static float __saturatef(float x) { return x > 0.f ? (x < 1.f ? x : 1.f) : 0.f; }
static float __fdividef(float a, float b) { return a / b; }
static float rsqrtf(float x) { return (float)(1.0 / std::sqrt((double)x)) * g_rsqrt; }
template <class R> static R dot3(const R *a, const R *b) { return std::fma(a[2], b[2], std::fma(a[1], b[1], a[0] * b[0])); }

SOURCE

typedef long double Q;
static Q dist2(const Q *r) { return r[0] * r[0] + r[1] * r[1] + r[2] * r[2]; }
static Q clamp(Q x) { return x > 0 ? (x < 1 ? x : 1) : 0; }
static Q point_seg(const Q *X, const Q *T, const Q *H) {
  Q u[3], w[3], a = 0, b = 0;
  for (int k = 0; k < 3; ++k) { u[k] = H[k] - T[k]; w[k] = X[k] - T[k]; a += u[k] * u[k]; b += u[k] * w[k]; }
  const Q s = a > 0 ? clamp(b / a) : 0;
  Q r[3];
  for (int k = 0; k < 3; ++k) r[k] = w[k] - s * u[k];
  return dist2(r);
}
static Q seg_seg(const Q *H, const Q *T, const Q *K, const Q *S) {
  Q best = std::fmin(std::fmin(point_seg(H, S, K), point_seg(T, S, K)), std::fmin(point_seg(K, T, H), point_seg(S, T, H)));
  Q u[3], v[3], w[3], a = 0, b = 0, c = 0, d = 0, e = 0;
  for (int k = 0; k < 3; ++k) {
    u[k] = H[k] - T[k]; v[k] = K[k] - S[k]; w[k] = T[k] - S[k];
    a += u[k] * u[k]; b += u[k] * v[k]; c += v[k] * v[k]; d += u[k] * w[k]; e += v[k] * w[k];
  }
  const Q den = a * c - b * b;
  if (den > 0) {
    const Q s = clamp((b * e - c * d) / den), t = clamp((a * e - b * d) / den);
    Q r[3];
    for (int k = 0; k < 3; ++k) r[k] = w[k] + s * u[k] - t * v[k];
    best = std::fmin(best, dist2(r));
  }
  return std::sqrt(best);
}
static Q point_tri(const Q V[3][3], const Q *X) {
  Q best = std::fmin(point_seg(X, V[0], V[1]), std::fmin(point_seg(X, V[1], V[2]), point_seg(X, V[2], V[0])));
  Q a = 0, b = 0, c = 0, d = 0, e = 0, E[3], F[3], D[3];
  for (int k = 0; k < 3; ++k) {
    E[k] = V[1][k] - V[0][k]; F[k] = V[2][k] - V[0][k]; D[k] = X[k] - V[0][k];
    a += E[k] * E[k]; b += E[k] * F[k]; c += F[k] * F[k]; d += E[k] * D[k]; e += F[k] * D[k];
  }
  const Q den = a * c - b * b, s = (c * d - b * e) / den, t = (a * e - b * d) / den;
  if (den > 0 && s >= 0 && t >= 0 && s + t <= 1) {
    Q r[3];
    for (int k = 0; k < 3; ++k) r[k] = D[k] - s * E[k] - t * F[k];
    best = std::fmin(best, dist2(r));
  }
  return std::sqrt(best);
}

int main(int argc, char **argv) {
  std::mt19937_64 gen(17);
  std::normal_distribution<double> N;
  std::uniform_real_distribution<double> U(0, 1);
  const int n = atoi(argv[1]);
  Q seg_worst = 0, face_worst = 0, extent_worst = 0;
  for (int it = 0; it < n; ++it) {
    double A[3][3], B[3][3];
    const double size = std::pow(10.0, 4 * U(gen) - 2), gap = std::pow(10.0, 6 * U(gen) - 6) * size;
    const double far = it % 3 ? 0.0 : 1e3 * size, thin = it % 5 ? 1.0 : std::pow(10.0, -6 * U(gen));
    double o[3] = {N(gen) * far, N(gen) * far, N(gen) * far}, g[3] = {N(gen) * gap, N(gen) * gap, N(gen) * gap};
    for (int v = 0; v < 3; ++v)
      for (int k = 0; k < 3; ++k) {
        A[v][k] = o[k] + size * N(gen) * (k == 2 ? thin : 1.0);
        B[v][k] = o[k] + g[k] + size * N(gen) * (k == 2 ? thin : 1.0);
      }
    if (it % 7 == 0)  // B close to A's plane, or touching it at a vertex
      for (int k = 0; k < 3; ++k) B[it % 3][k] = A[(it / 7) % 3][k] + g[k];
    float a[3][3], b[3][3], L = 0.f;
    double LL = 0;
    Q QA[3][3], QB[3][3];
    for (int k = 0; k < 3; ++k) {
      float lo = 0.f, hi = 0.f;
      double dlo = A[0][k], dhi = A[0][k];
      for (int v = 0; v < 3; ++v) {
        a[v][k] = v ? (float)(A[v][k] - A[0][k]) : 0.f;
        b[v][k] = (float)(B[v][k] - A[0][k]);
        lo = std::fmin(lo, std::fmin(a[v][k], b[v][k]));
        hi = std::fmax(hi, std::fmax(a[v][k], b[v][k]));
        dlo = std::fmin(dlo, std::fmin(A[v][k], B[v][k]));
        dhi = std::fmax(dhi, std::fmax(A[v][k], B[v][k]));
        QA[v][k] = A[v][k];
        QB[v][k] = B[v][k];
      }
      L = std::fmax(L, hi - lo);
      LL = std::fmax(LL, dhi - dlo);
    }
    extent_worst = std::fmax(extent_worst, std::fabs((Q)L - LL) / (LL * kU32));
    const Q unit = (Q)kU32 * L;
    for (float e : {1.f - 2.4e-7f, 1.f, 1.f + 2.4e-7f}) {
      g_rsqrt = e;
      delta_edge(a, b, QA, QB, unit, seg_worst);
      delta_face(a, b, QA, QB, unit, face_worst);
    }
  }
  std::printf("%.3Lf %.3Lf %.3Lf\n", seg_worst, face_worst, extent_worst);
}
"""

CALLS = r"""
typedef long double Q;
static Q seg_seg(const Q *, const Q *, const Q *, const Q *);
static Q point_tri(const Q V[3][3], const Q *);
static void delta_edge(float a[3][3], float b[3][3], Q A[3][3], Q B[3][3], Q unit, Q &worst) {
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      float lb;
      seg_seg_lb(a[(i + 1) % 3], edge_frame(a[i], a[(i + 1) % 3]), b[(j + 1) % 3], edge_frame(b[j], b[(j + 1) % 3]), lb);
      const Q over = lb - seg_seg(A[i], A[(i + 1) % 3], B[j], B[(j + 1) % 3]);
      if (over > worst * unit) worst = over / unit;
    }
}
static void delta_face(float a[3][3], float b[3][3], Q A[3][3], Q B[3][3], Q unit, Q &worst) {
  for (int j = 0; j < 6; ++j) {
    float lb;
    if (j < 3) pt_tri_lb(a[0], tri_frame(a), b[j], 0.f, lb);
    else pt_tri_lb(b[0], tri_frame(b), a[j - 3], 0.f, lb);
    const Q over = lb - (j < 3 ? point_tri(A, B[j]) : point_tri(B, A[j - 3]));
    if (over > worst * unit) worst = over / unit;
  }
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_the_band_covers_the_rounding_with_room(tmp_path):
    text = (CSRC / "tri_cert.cuh").read_text()
    source = text[text.index("constexpr float kU32"):text.index("// A vertex (0..2) of A or B")]
    source = re.sub(r"#pragma unroll[^\n]*", "", source)
    src, exe = tmp_path / "band.cpp", tmp_path / "band"
    src.write_text(HARNESS.replace("SOURCE", source + CALLS))
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), "300000"], check=True, capture_output=True, text=True).stdout
    seg, face, extent = (float(x) for x in out.split())
    assert 0.0 < seg <= 42.0 and 0.0 < face <= 42.0, out
    assert extent <= 3.0, out


def test_a_float_exceeds_a_double_when_it_exceeds_the_double_rounded_down():
    rng = np.random.default_rng(3)
    f = np.concatenate([rng.normal(size=100_000), 10.0 ** rng.uniform(-45, 38, 100_000),
                        [0.0, -0.0, np.inf, -np.inf, np.nan, 1e-45, 3.4028235e38]]).astype(np.float32)
    for d in (f.astype(np.float64), np.nextafter(f.astype(np.float64), np.inf),
              np.nextafter(f.astype(np.float64), -np.inf), f.astype(np.float64) * 1.0000001, np.full(f.shape, 1e308)):
        with np.errstate(over="ignore", invalid="ignore"):
            r = d.astype(np.float32)
            r = np.where(r.astype(np.float64) > d, np.nextafter(r, np.float32(-np.inf)), r)
        assert np.array_equal(f > r, f.astype(np.float64) > d)
