"""The short division and square root of csrc/ct_fp64.cuh round correctly whatever FP32 estimate the
hardware gives within its documented error (2 units in the last place of __fdividef and rsqrtf): the
source compiled for the host, with estimates moved by -2 .. 2 units, against the host's / and sqrt.
"""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
HARNESS = r"""
#include <stdio.h>
#include "fp64_scalars.h"
#define __device__
#define __forceinline__ inline
static long long __double_as_longlong(double x) { long long v; memcpy(&v, &x, 8); return v; }
static double __longlong_as_double(long long x) { double v; memcpy(&v, &x, 8); return v; }
static int __float_as_int(float x) { int v; memcpy(&v, &x, 4); return v; }
static float __int_as_float(int x) { float v; memcpy(&v, &x, 4); return v; }
static int moved = 0;
static float move(float x) { return __int_as_float(__float_as_int(x) + moved); }
static float __fdividef(float a, float b) { return move(a / b); }
static float estimate_rsqrt(float x) { return move((float)(1.0 / sqrt((double)x))); }
#define rsqrtf estimate_rsqrt
#include "ct_fp64.cuh"
int main() {
    std::vector<double> n, d, x;
    fp64_cases::divisions(100000, n, d);
    fp64_cases::roots(100000, x);
    long bad_q = 0, bad_r = 0;
    for (moved = -2; moved <= 2; ++moved) {
        for (size_t i = 0; i < n.size(); ++i) bad_q += !fp64_cases::same(ct_fp64::div_rn(n[i], d[i]), n[i] / d[i]);
        for (double v : x) bad_r += !fp64_cases::same(ct_fp64::sqrt_rn(v), sqrt(v));
    }
    printf("%zu %ld %zu %ld\n", n.size(), bad_q, x.size(), bad_r);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_correctly_rounded_for_every_estimate(tmp_path):
    src = tmp_path / "scalars.cpp"
    src.write_text(HARNESS)
    exe = tmp_path / "scalars"
    # (no contraction: only the fma calls of the source may be fused)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-x", "c++", "-I", str(ROOT / "tests"), "-I",
                    str(ROOT / "chemtensor_mojo_gb300" / "csrc"), str(src), "-o", str(exe), "-lm"], check=True)
    cases_q, bad_q, cases_r, bad_r = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert cases_q > 1000000 and cases_r > 400000
    assert (bad_q, bad_r) == (0, 0)
