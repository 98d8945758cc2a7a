"""The table-driven logarithm against the one through CUDA's log in double, over
the positive normal floats in steps and around 1, and the same bits for zero,
subnormals, infinity and NaN.  Both round a double once.  The doubles are within
2.3e-16 (series) plus two roundings, 2.2e-16, of each other, and a float rounds
differently only if its logarithm lies that near the middle of two floats, which
are at least 2^-24 apart, relatively: a share of 2 * 4.5e-16 / 6e-8 = 1.5e-8, and by
one unit in the last place."""
import ctypes
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "common.cuh"
__global__ void k(unsigned lo, unsigned hi, unsigned step, unsigned* out) {
  __shared__ __align__(16) double2 t[lre::LOG_TAB_N];
  lre::log_tab_fill(t);
  __syncthreads();
  for (unsigned long long b = lo + (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) * step; b < hi;
       b += (unsigned long long)gridDim.x * blockDim.x * step) {
    const float x = __int_as_float((int)b);
    const int p = __float_as_int(lre::log_tab(t, x)), q = __float_as_int(lre::log_cr(x));
    if (p != q) {
      atomicAdd(out, 1u);
      atomicMax(out + 1, (unsigned)abs(p - q));
    }
  }
}
extern "C" int run(unsigned lo, unsigned hi, unsigned step, unsigned* host) {
  unsigned* d;
  if (cudaMalloc(&d, 8) != cudaSuccess || cudaMemset(d, 0, 8) != cudaSuccess) return 1;
  k<<<592, 256>>>(lo, hi, step, d);
  const int rc = cudaMemcpy(host, d, 8, cudaMemcpyDeviceToHost) != cudaSuccess;
  cudaFree(d);
  return rc;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("log_table")
    (d / "k.cu").write_text(SRC)
    subprocess.run([nvcc, "-std=c++17", "-O3", "--fmad=false", "-gencode", "arch=compute_100a,code=sm_100a", "-shared",
                    "-Xcompiler", "-fPIC", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "libraw_enhanced_b200", "csrc"), str(d / "k.cu"), "-o", str(d / "k.so")],
                   check=True)
    return ctypes.CDLL(str(d / "k.so"))


@pytest.mark.parametrize("lo,hi,step", [
    (0x00800000, 0x7f800000, 7),  # all normals, one of seven
    (0x3f7f0000, 0x3f810000, 1),  # the intervals at 1, where the logarithm is small
    (0x3f330000 - 70000, 0x3f330000 + 70000, 1), (0x3fb30000 - 70000, 0x3fb30000 + 70000, 1),  # the ends of m's range
    (0x00000000, 0x00800000, 5), (0x7f800000, 0x7f800400, 1), (0x80000000, 0x80000400, 1)])  # not normal
def test_log_table(lib, lo, hi, step):
    out = (ctypes.c_uint * 2)()
    assert lib.run(lo, hi, step, out) == 0
    normal = 0x00800000 <= lo < 0x7f800000
    share = 1.5e-8 * ((hi - lo) / step)
    assert out[0] <= (max(1, share) if normal else 0)
    assert out[1] <= (1 if out[0] else 0)
