"""The fused kernels' GELU has the bits of the GEMM kernels' for every float.

The fused kernels round GELU to BF16 from an approximation with an error bound, and fall back to
the function itself where the bound does not decide the rounding.  All 2^32 arguments, in pairs with a
neighbour of another magnitude, are compared on the GPU with the function.
"""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "se2dr_fork_gb300", "csrc")
SOURCE = r"""
#include "se2nn_rows.cuh"
#include <cstdio>
__global__ void check(unsigned long long *out)
{
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < (1ull << 32);
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const float x = __uint_as_float((unsigned)i), y = __uint_as_float((unsigned)i * 2654435761u);
    if (nnk::gelu_pack(x, y) != nnk::pack_bf16(nnk::gelu_f(x), nnk::gelu_f(y))) atomicAdd(out, 1ull);
  }
}
int main()
{
  unsigned long long *d, n = ~0ull;
  cudaMalloc(&d, sizeof n);
  cudaMemset(d, 0, sizeof n);
  check<<<608, 256>>>(d);
  if (cudaMemcpy(&n, d, sizeof n, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  printf("%llu\n", n);
  return 0;
}
"""


@pytest.mark.gpu
def test_every_float(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, exe = tmp_path / "gelu.cu", tmp_path / "gelu"
    src.write_text(SOURCE)
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_103a,code=sm_103a", "-I", CSRC,
                    "-o", str(exe), str(src)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout.strip() == "0"
