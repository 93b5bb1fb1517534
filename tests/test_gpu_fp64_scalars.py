"""The short division and square root of csrc/ct_fp64.cuh against CUDA's / and sqrt on the device, bit for
bit, over the hard operands of fp64_scalars.h and a million random ones.
"""
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent
HARNESS = r"""
#include <stdio.h>
#include <cuda_runtime.h>
#include "fp64_scalars.h"
#include "ct_fp64.cuh"
__global__ void run(const double* n, const double* d, size_t nq, const double* x, size_t nr, unsigned long long* bad) {
    auto differs = [](double a, double b) {
        return __double_as_longlong(a) != __double_as_longlong(b) && !(isnan(a) && isnan(b));
    };
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nq; i += (size_t)gridDim.x * blockDim.x)
        if (differs(ct_fp64::div_rn(n[i], d[i]), n[i] / d[i])) atomicAdd(bad, 1ull);
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nr; i += (size_t)gridDim.x * blockDim.x)
        if (differs(ct_fp64::sqrt_rn(x[i]), sqrt(x[i]))) atomicAdd(bad + 1, 1ull);
}
int main() {
    std::vector<double> n, d, x;
    fp64_cases::divisions(250000, n, d);
    fp64_cases::roots(250000, x);
    double *dn, *dd, *dx;
    unsigned long long *db, bad[2] = {0, 0};
    if (cudaMalloc(&dn, n.size() * 8) || cudaMalloc(&dd, d.size() * 8) || cudaMalloc(&dx, x.size() * 8) || cudaMalloc(&db, 16)) return 1;
    cudaMemcpy(dn, n.data(), n.size() * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(dd, d.data(), d.size() * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(dx, x.data(), x.size() * 8, cudaMemcpyHostToDevice);
    cudaMemset(db, 0, 16);
    run<<<304, 256>>>(dn, dd, n.size(), dx, x.size(), db);
    if (cudaMemcpy(bad, db, 16, cudaMemcpyDeviceToHost)) return 1;
    printf("%zu %llu %zu %llu\n", n.size(), bad[0], x.size(), bad[1]);
}
"""


def test_bits_of_the_cuda_operators(tmp_path):
    from chemtensor_mojo_gb300 import build
    src = tmp_path / "scalars.cu"
    src.write_text(HARNESS)
    exe = tmp_path / "scalars"
    subprocess.run([build._nvcc(), "-O2", "-std=c++17", *build.ARCH, "-I", str(ROOT / "tests"), "-I",
                    str(ROOT / "chemtensor_mojo_gb300" / "csrc"), str(src), "-o", str(exe)], check=True)
    cases_q, bad_q, cases_r, bad_r = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert cases_q > 2500000 and cases_r > 1000000
    assert (bad_q, bad_r) == (0, 0)
