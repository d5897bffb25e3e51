"""The packed correctly rounded reciprocal, quotient and square root of the Smagorinsky collision against
CUDA's own IEEE operations, bit for bit: every significand for the reciprocal, every significand of two
binades for the root, 2^26 quotients."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import cells_b200.geometry as g
from cells_b200 import Solver3D
from cells_b200.rng import perturbed_rest3

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cstdio>
#include "rn2.cuh"
__device__ unsigned mix(unsigned v) { v ^= v >> 16; v *= 0x7feb352du; v ^= v >> 15; v *= 0x846ca68bu; return v ^ (v >> 16); }
__device__ float number(unsigned m, int e) { return __int_as_float((int)((m & 0x7fffffu) | ((unsigned)(e + 127) << 23))); }
__global__ void check(int what, int exponent, unsigned long long* bad) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  const float2 x = make_float2(number(i, exponent), number(i, exponent + 1));
  float2 got, want;
  if (what == 0) {
    got = cells::rn_rcp2(x);
    want = make_float2(__frcp_rn(x.x), __frcp_rn(x.y));
  } else if (what == 1) {
    got = cells::rn_sqrt2(x);
    want = make_float2(__fsqrt_rn(x.x), __fsqrt_rn(x.y));
  } else {
    const unsigned k = mix(i * 2654435761u + (unsigned)exponent);
    const float2 a = make_float2(number(k, (int)(k >> 27) - 16), number(mix(k), exponent / 2));
    got = cells::rn_div2(a, x, cells::rn_rcp2(x));
    want = make_float2(__fdiv_rn(a.x, x.x), __fdiv_rn(a.y, x.y));
  }
  if (__float_as_int(got.x) != __float_as_int(want.x) || __float_as_int(got.y) != __float_as_int(want.y))
    atomicAdd(bad, 1ull);
}
int main() {
  unsigned long long *bad, host = 0;
  if (cudaMalloc(&bad, 8) != cudaSuccess) return 2;
  int failed = 0;
  for (int what = 0; what < 3; what++) {
    for (int e = -40; e <= 40; e += 16) {
      cudaMemset(bad, 0, 8);
      check<<<(1 << 23) / 256, 256>>>(what, e, bad);
      if (cudaMemcpy(&host, bad, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
      if (host) printf("operation %d exponent %d: %llu differ\n", what, e, host);
      failed |= host != 0;
    }
  }
  return failed;
}
"""


def test_bits_equal_ieee(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    assert os.path.exists(nvcc)
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cells_b200", "csrc")
    src, exe = tmp_path / "check.cu", tmp_path / "check"
    src.write_text(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-I", csrc, "-ccbin", "/usr/bin/g++",
                    "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout


def solver(**kw):
    W, H, D = 40, 14, 12
    s = Solver3D.create(W, H, D, **dict(dict(tau=0.56, uIn=0.05, smagorinsky=0.1, forceEvery=0), **kw))
    sdf = g.empty_sdf3(W, H, D)
    g.add_sphere(sdf, W, H, D, 12, 7, 6, 2.6)
    s.setSdf(sdf)
    s.initField(perturbed_rest3(W, H, D, 1e-3, ux=0.05))
    return s


def test_switching_smagorinsky_rebuilds_the_rates():
    a, b = solver(smagorinsky=0.0), solver()
    a.setSmagorinsky(0.1)
    for s in (a, b):
        s.encodeSteps(7)
    assert np.array_equal(a.readPopulations(), b.readPopulations())
    for s in (a, b):
        s.setSmagorinsky(0.0)
        s.encodeSteps(7)
    assert np.array_equal(a.readPopulations(), b.readPopulations())


# Relaxation times that round to 1/2 in f32 leave the packed operations' range; the fast and the exact build
# differ by at most 40 roundings of the largest population per step, which relaxation does not amplify in 12.
@pytest.mark.parametrize("tau", [0.5 + 1e-9, 0.5000005, 0.51, 2.0])
@pytest.mark.parametrize("lam", [None, 0.0, 0.25])
def test_relaxation_times_next_to_one_half(tau, lam):
    kw = {} if lam is None else {"lambda_": lam}
    a, b = solver(tau=tau, **kw), solver(tau=tau, exactArithmetic=True, **kw)
    for s in (a, b):
        s.encodeSteps(12)
    x, y = a.readPopulations(), b.readPopulations()
    assert np.all(np.isfinite(x))
    assert np.max(np.abs(x - y)) <= 12 * 40 * 6e-8 * np.max(np.abs(y))
