"""The scalar and the packed forms of the network's activation round alike (no GPU).

The layer-by-layer kernels use gelu and gelu_grad, the fused ones gelu2 and gelu_grad2
(delta_b200/csrc/mlp.cuh). Both are compiled here for the host, with the packed operations
lane by lane, no contraction, and tanhf for the hardware's tanh, and compared bit for bit: a
multiply-add that only one of them writes out would show.
"""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

SRC = Path(__file__).resolve().parents[1] / "delta_b200" / "csrc" / "mlp.cuh"

HARNESS = r"""
#include <math.h>
#include <cstdint>
#include <cstdio>
#include <cstring>
#define __device__
#define __forceinline__ inline
struct float2 { float x, y; };
static float2 make_float2(float x, float y) { return {x, y}; }
static float2 __fmul2_rn(float2 a, float2 b) { return {a.x * b.x, a.y * b.y}; }
static float2 __fadd2_rn(float2 a, float2 b) { return {a.x + b.x, a.y + b.y}; }
static float2 __ffma2_rn(float2 a, float2 b, float2 c) { return {fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)}; }
static float tanh_hw(float x) { return tanhf(x); }
SOURCE
static bool same(float a, float b) { return memcmp(&a, &b, 4) == 0 || (a != a && b != b); }
int main() {
  long bad = 0, n = 0;
  for (uint64_t u = 0; u < 1ull << 32; u += 1021, ++n) {
    const uint32_t bits = (uint32_t)u;
    float x;
    memcpy(&x, &bits, 4);
    const float2 v = make_float2(x, -x), g = gelu2(v), d = gelu_grad2(v);
    bad += !same(g.x, gelu(x)) + !same(g.y, gelu(-x)) + !same(d.x, gelu_grad(x)) + !same(d.y, gelu_grad(-x));
  }
  printf("%ld of %ld\n", bad, n);
  return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_packed_and_scalar_forms_round_alike(tmp_path):
    text = SRC.read_text()
    source = text[text.index("constexpr float kGeluK"):text.index("__device__ __forceinline__ uint32_t pack_bf16(float2 v)")]
    assert all(re.search(r"\b" + f + r"\(float", source) for f in ("gelu", "gelu_grad", "gelu2", "gelu_grad2"))
    src, exe = tmp_path / "gelu.cpp", tmp_path / "gelu"
    src.write_text(HARNESS.replace("SOURCE", source))
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
