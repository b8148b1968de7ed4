"""The device forms of the reproducible exp and log (csrc/portable_math.h) give
the host's bits: the logarithm's quotient for every value it can have, the
functions over a stride of all single-precision numbers."""
import pathlib
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parents[1]

SOURCE = r"""
#include <cstdio>
#include <vector>
#include <math.h>
#include "portable_math.h"
__global__ void Quotients(unsigned first, unsigned count, unsigned *wrong) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count)
    return;
  const float f = __uint_as_float(first + i) - 1.0f, b = 2.0f + f;
  if (__float_as_uint(thmm_log_quotient(f, b)) != __float_as_uint(__fdiv_rn(f, b)))
    atomicAdd(wrong, 1u);
}
__global__ void Values(unsigned stride, unsigned count, float *logs, float *exps) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count)
    return;
  const float x = __uint_as_float(i * stride);
  logs[i] = thmm_logf(x);
  exps[i] = thmm_expf_nonpositive(x);
}
static bool Same(float a, float b) { return thmm_f2u(a) == thmm_f2u(b) || (a != a && b != b); }
int main() {
  const unsigned first = 0x3f3504f4u, count = 0x3fb504f4u - 0x3f3504f4u;
  unsigned *wrong, quotients = 1;
  cudaMalloc(&wrong, 4);
  cudaMemset(wrong, 0, 4);
  Quotients<<<(count + 255) / 256, 256>>>(first, count, wrong);
  cudaMemcpy(&quotients, wrong, 4, cudaMemcpyDeviceToHost);
  const unsigned stride = 509, n = 0xffffffffu / stride;
  float *logs, *exps;
  cudaMalloc(&logs, n * 4ull);
  cudaMalloc(&exps, n * 4ull);
  Values<<<(n + 255) / 256, 256>>>(stride, n, logs, exps);
  std::vector<float> l(n), e(n);
  cudaMemcpy(l.data(), logs, n * 4ull, cudaMemcpyDeviceToHost);
  cudaMemcpy(e.data(), exps, n * 4ull, cudaMemcpyDeviceToHost);
  unsigned values = 0;
  for (unsigned i = 0; i < n; ++i) {
    const float x = thmm_u2f(i * stride);
    values += !Same(l[i], thmm_logf(x)) || !Same(e[i], thmm_expf_nonpositive(x));
  }
  std::printf("%u quotients, %u values differ, %s\n", quotients, values,
              cudaGetErrorString(cudaGetLastError()));
  return quotients != 0 || values != 0 || cudaGetLastError() != cudaSuccess;
}
"""


def test_device_functions_match_the_host(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    source = tmp_path / "values.cu"
    source.write_text(SOURCE)
    binary = tmp_path / "values"
    subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-Xcompiler", "-ffp-contract=off",
                    f"-I{ROOT / 'parallel_tree_hmm_gb300' / 'csrc'}", str(source), "-o",
                    str(binary)], check=True)
    result = subprocess.run([str(binary)], capture_output=True, text=True, timeout=300)
    assert result.returncode == 0, result.stdout
