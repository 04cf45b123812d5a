"""A bounded wait that ran out is reported whichever lane it ran out for.

Every lane of a warp polls a barrier for itself, so the limit can end the wait
of any of them alone.  No wait is made to run out here: the flags are given.
"""
import ctypes
import subprocess

import numpy as np
import pytest

from fv3d_gb300 import build as fvbuild

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "fv_device.cuh"
__global__ void report(const unsigned* lanes, int* err) {
  fv::report_late(lanes[blockIdx.x] >> (threadIdx.x & 31) & 1u, err + blockIdx.x);
}
extern "C" int run(int n, const unsigned* lanes, int* err) {
  unsigned* d = nullptr;
  if (cudaMalloc(&d, 2 * n * sizeof(int)) != cudaSuccess) return 1;
  cudaMemcpy(d, lanes, n * sizeof(int), cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, err, n * sizeof(int), cudaMemcpyHostToDevice);
  report<<<n, 32>>>(d, reinterpret_cast<int*>(d + n));
  const cudaError_t e = cudaMemcpy(err, d + n, n * sizeof(int), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
"""


def test_any_lane(tmp_path):
    src, so = str(tmp_path / "late.cu"), str(tmp_path / "late.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.check_call([fvbuild._nvcc(), *fvbuild.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-I",
                           fvbuild.CSRC, "-I", fvbuild.INCLUDE, "-shared", "-o", so, src])
    lanes = np.array([0, *(1 << k for k in range(32)), 0xffffffff, 0x80000002], np.uint32)
    err = np.arange(lanes.size, dtype=np.int32) % 2  # a flag that is set already stays
    want = err | np.where(lanes != 0, 2, 0)
    run = ctypes.CDLL(so).run
    assert run(lanes.size, lanes.ctypes.data_as(ctypes.c_void_p), err.ctypes.data_as(ctypes.c_void_p)) == 0
    np.testing.assert_array_equal(err, want)
