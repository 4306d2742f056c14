"""The reciprocal and quotient of the loss and adjoint kernels (`rcp_newton`,
`quot_newton`, quantom_b200/csrc/physmath.cuh) against IEEE division, bit for
bit: the reciprocal at every significand, the quotient at four numerators each,
over the powers of two that squared and plain pair distances take (0.004 to
16).  A small program compiled from the header and run on the GPU."""
import shutil
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHECK = r"""
#include <cstdio>
#include "physmath.cuh"
__global__ void compare(unsigned long long* bad, int e) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (1u << 23)) return;
    const float x = ldexpf(1.f + i * 0x1p-23f, e);
    if (lima::rcp_newton(x) != 1.f / x) atomicAdd(&bad[0], 1ull);
    unsigned h = i * 2654435761u;
    for (int t = 0; t < 4; t++) {
        h = h * 1664525u + 1013904223u;
        const float g = ldexpf((h & 1u ? -1.f : 1.f) * (1.f + (h >> 9) * 0x1p-23f), (int)((h >> 1) % 20u) - 10);
        if (lima::quot_newton(g, x) != g / x) atomicAdd(&bad[1], 1ull);
    }
    if (lima::quot_newton(0.f, x) != 0.f) atomicAdd(&bad[1], 1ull);
}
int main() {
    unsigned long long* bad = nullptr;
    if (cudaMalloc(&bad, 2 * sizeof(*bad)) != cudaSuccess || cudaMemset(bad, 0, 2 * sizeof(*bad)) != cudaSuccess) return 2;
    for (int e = -8; e <= 3; e++) compare<<<(1 << 23) / 256, 256>>>(bad, e);
    unsigned long long h[2] = {1, 1};
    if (cudaMemcpy(h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    printf("%llu %llu\n", h[0], h[1]);
    return 0;
}
"""


def test_reciprocal_and_quotient_round_correctly(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not shutil.which(nvcc):
        pytest.skip("nvcc not found")
    src = tmp_path / "check.cu"
    src.write_text(CHECK)
    exe = tmp_path / "check"
    subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", f"-I{ROOT / 'include'}",
                    f"-I{ROOT / 'quantom_b200' / 'csrc'}", str(src), "-o", str(exe)],
                   check=True, capture_output=True, timeout=600)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and out.stdout.split() == ["0", "0"], out.stdout
