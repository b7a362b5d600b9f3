"""The acceptance test that takes the hardware logarithm first (neglog_gap): over
every uniform there is, its distance from the exact variate stays within the
tolerance beyond which the kernels take its sign for the decision."""
import ctypes as C
import importlib.util
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

SOURCE = r"""
#include <cuda_runtime.h>
#include "oj_device.cuh"
// out: the largest |gap - (x - neglog)| in units of 2^-40, and the decisions it gets wrong
__global__ void check(unsigned long long* out) {
  unsigned long long worst = 0, wrong = 0;
  for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < 1u << 23; k += gridDim.x * blockDim.x) {
    const unsigned word = (k << 9) | (k & 511u);
    const float exact = ojd::neglog(word);
    for (int d = -40; d <= 40; ++d) {
      const float x = exact + d * 0x1p-18f;
      const float t = ojd::neglog_gap(x, word);
      const unsigned long long dev = (unsigned long long)(fabs((double)t - ((double)x - (double)exact)) * 0x1p40);
      worst = dev > worst ? dev : worst;
      if (fabsf(t) > ojd::kNegLogTol && (t < 0.0f) != (x < exact)) ++wrong;
    }
  }
  atomicMax(out, worst);
  atomicAdd(out + 1, wrong);
}
extern "C" int run(double* worst, unsigned long long* wrong) {
  unsigned long long *d = nullptr, h[2];
  cudaError_t e = cudaMalloc(&d, sizeof h);
  if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof h);
  if (e == cudaSuccess) {
    check<<<592, 256>>>(d);
    e = cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost);
  }
  *worst = h[0] * 0x1p-40;
  *wrong = h[1];
  cudaFree(d);
  return e;
}
"""


def test_hardware_logarithm_stays_within_its_tolerance(tmp_path):
    spec = importlib.util.spec_from_file_location("_recipe", os.path.join(HERE, "..", "openjij_b200", "build.py"))
    recipe = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(recipe)
    src, lib = tmp_path / "gap.cu", tmp_path / "gap.so"
    src.write_text(SOURCE)
    subprocess.run([recipe.NVCC] + recipe.ARCH + recipe.NVCC_FLAGS + ["-shared", str(src), "-o", str(lib)], check=True)
    worst, wrong = C.c_double(), C.c_ulonglong()
    assert C.CDLL(str(lib)).run(C.byref(worst), C.byref(wrong)) == 0
    assert wrong.value == 0
    assert worst.value <= 2.0 ** -16
