"""The integer-pipe conversions and splits against the hardware's, value by
value: the edges of the FP32 range, denormals, ties, mantissa carries, zeros,
infinities and NaN."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "wf_step_common.cuh"
using namespace wf;
__device__ bool same(float a, float b) { return a == b || (isnan(a) && isnan(b)); }
__device__ bool same(double a, double b) { return a == b || (isnan(a) && isnan(b)); }
__global__ void k_compare(const double* v, int n, unsigned* bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = v[i];
  const float f = __double2float_rn(x);
  unsigned m = 0;
  if (!same(d2f(x), f)) m |= 1;
  if (!same(f2d(f), (double)f)) m |= 2;
  const float lo = __double2float_rn(x - (double)f);
  float h, l;
  ff_split(x, h, l);
  if (!same(h, f) || !same(l, lo)) m |= 4;
  const double t[3] = {x, -x, v[n - 1 - i]};
  float h3[3], l3[3];
  ff_split3(t, h3, l3);
  for (int d = 0; d < 3; ++d) {
    const float g = __double2float_rn(t[d]);
    if (!same(h3[d], g) || !same(l3[d], __double2float_rn(t[d] - (double)g))) m |= 8;
  }
  bad[i] = m;
}
extern "C" int compare(const double* host, int n, unsigned* out) {
  double* v = nullptr;
  unsigned* bad = nullptr;
  if (cudaMalloc(&v, n * sizeof(double)) != cudaSuccess || cudaMalloc(&bad, n * sizeof(unsigned)) != cudaSuccess) return 1;
  cudaMemcpy(v, host, n * sizeof(double), cudaMemcpyHostToDevice);
  k_compare<<<(n + 127) / 128, 128>>>(v, n, bad);
  cudaMemcpy(out, bad, n * sizeof(unsigned), cudaMemcpyDeviceToHost);
  cudaFree(v);
  cudaFree(bad);
  return (int)cudaGetLastError();
}
"""


def _values():
    rng = np.random.default_rng(11)
    m = np.concatenate([[1.0, 2.0 - 2.0 ** -52, 2.0 - 2.0 ** -24, 2.0 - 2.0 ** -23, 1.0 + 2.0 ** -24, 1.0 + 3 * 2.0 ** -24,
                         1.0 + 2.0 ** -24 + 2.0 ** -52, 1.0 + 2.0 ** -52, 1.5, 1.0 + 2.0 ** -29],
                        1.0 + rng.random(40)])
    e = np.concatenate([np.arange(-1074, -1060), np.arange(-160, 135), [-1022, -500, 500, 1023]]).astype(int)
    v = np.ldexp(m[None, :], e[:, None]).ravel()
    v = np.concatenate([v, [0.0, np.inf, np.nan, np.finfo(np.float32).max, np.finfo(np.float32).tiny]])
    v = np.concatenate([v, -v])
    return np.ascontiguousarray(v[rng.permutation(len(v))])


def test_conversions_and_splits_give_the_hardware_values(tmp_path):
    src, lib = tmp_path / "compare.cu", tmp_path / "libcompare.so"
    src.write_text(SOURCE)
    r = subprocess.run([ge._nvcc(), *ge.NVCC_FLAGS, "-I", ge.CSRC, "-shared", "-o", os.fspath(lib), os.fspath(src)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    v = _values()
    bad = np.full(len(v), 0xFFFF, dtype=np.uint32)
    f = ctypes.CDLL(os.fspath(lib)).compare
    f.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
    assert f(v.ctypes.data, len(v), bad.ctypes.data) == 0
    for bit, name in ((1, "d2f"), (2, "f2d"), (4, "ff_split"), (8, "ff_split3")):
        at = np.nonzero(bad & bit)[0]
        assert len(at) == 0, (name, len(at), [float(q).hex() for q in v[at[:5]]])
