"""A wait on a phase that nothing completes ends after a fraction of a second, and the other waits of its CTA give up with it."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ojasx-vector-24x96_b200", "csrc")

SOURCE = r"""
#include <cstdio>
#include "common.cuh"
__global__ void waits(int* out) {
    __shared__ unsigned long long bars[2];
    __shared__ int gone;
    const unsigned b = static_cast<unsigned>(__cvta_generic_to_shared(bars)), g = static_cast<unsigned>(__cvta_generic_to_shared(&gone));
    if (threadIdx.x == 0) {
        gone = 0;
        for (int i = 0; i < 2; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b + 8 * i) : "memory");
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(b + 8) : "memory");
    }
    __syncthreads();
    int ended = 0;
    for (int i = 0; i < 100; ++i) ended += ojx::bar_wait(b, 0, g);        // nothing arrives there
    out[threadIdx.x] = ended + 2 * ojx::bar_wait(b + 8, 0, g) + 4 * gone;
}
int main() {
    int *d, h[64];
    cudaEvent_t t0, t1;
    cudaEventCreate(&t0); cudaEventCreate(&t1);
    cudaMalloc(&d, sizeof(h));
    cudaEventRecord(t0);
    waits<<<1, 64>>>(d);
    cudaEventRecord(t1);
    if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, t0, t1);
    for (int v : h) if (v != 6) { printf("status %d\n", v); return 1; }
    printf("%f\n", ms);
    return 0;
}
"""


def test_waits_end(cuda, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("needs nvcc")
    (tmp_path / "waits.cu").write_text(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", CSRC, "-o", str(tmp_path / "waits"), str(tmp_path / "waits.cu")],
                   check=True, timeout=120)
    run = subprocess.run([str(tmp_path / "waits")], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout + run.stderr
    assert 50 < float(run.stdout) < 1000      # 2^28 clocks once, not a hundred times
