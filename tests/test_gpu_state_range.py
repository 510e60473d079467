"""The float64 Euler kernels over the range of states that their fast fluxes
take (B200).

* Density times 2^a and velocity times 2^b scale every term of the right-hand
  side, the tangent and the adjoint by a power of two, so the scaled results are
  the unscaled ones to round-off (1e-12 as for the kernels' other comparisons),
  inside the checked range, at its ends and outside of it.  (HLL truncates a wave
  speed to an integer and does not scale.)
* The reciprocal and the two roots against the correctly rounded operations,
  2^-1000 to 2^1000 and at the floor of the squared speed: one unit in the last
  place, two for the reciprocal root (whose reference is rounded twice)."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from apollo_b200 import NodalDG2d
from apollo_b200.mesh import jittered_square
from golden_cases import rel_l2

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "apollo_b200", "csrc")
SCALES = [(399, 0), (401, 0), (-399, 0), (-401, 0), (510, 0), (-510, 0), (0, 199), (0, 201), (0, -199), (0, -201),
          (0, -230), (200, -340), (490, -490), (-490, 490), (380, -390), (-380, 390), (120, -40)]


def _solver(fields, flux, N):
    s = NodalDG2d(N, 0.5, {4: "eulerEqn2d", 5: "eulerEqn"}[fields], (1.4, 0.0, 0.0), jittered_square(5, seed=3),
                  numerical_flux=flux)
    rng = np.random.default_rng(N)
    U = rng.uniform(-0.1, 0.1, s.shape)
    U[..., 0] += 1.0
    U[..., 1] += 0.4
    U[9, :, 1:-1] = 0.0  # an element at rest
    U[..., -1] = 0.5 * (U[..., 1:-1] ** 2).sum(-1) / U[..., 0] + rng.uniform(2.3, 2.7, s.shape[:2])
    return s, U


def _scale(fields, a, b):
    return np.ldexp(1.0, np.array([a] + [a + b] * (fields - 2) + [a + 2 * b]))


@pytest.mark.parametrize("a,b", SCALES)
@pytest.mark.parametrize("fields,flux,N", [(4, "LF", 4), (5, "LF", 2), (4, "Roe", 3), (5, "Wave", 5), (5, "Roe", 4)])
def test_scaled_right_hand_side(fields, flux, N, a, b):
    s, U = _solver(fields, flux, N)
    r, sugg = s.step(0.0, 0.0, U)
    S = _scale(fields, a, b)
    rs, ss = s.step(0.0, 0.0, U * S)
    assert rel_l2(rs / S * np.ldexp(1.0, -b), r) <= 1e-12
    assert ss == pytest.approx(float(np.ldexp(sugg, -b)), rel=1e-13)


@pytest.mark.parametrize("a,b", SCALES)
@pytest.mark.parametrize("fields,N", [(4, 3), (5, 4)])
def test_scaled_derivatives(fields, N, a, b):
    s, U = _solver(fields, "LF", N)
    U[9, :, 1] += 0.3  # the speed of a state at rest has no derivative
    rng = np.random.default_rng(fields)
    v, w = rng.standard_normal(s.shape), rng.standard_normal(s.shape)
    S = _scale(fields, a, b)
    Sr = S * np.ldexp(1.0, b)
    assert rel_l2(s.rhs_jvp(0.0, U * S, v * S) / Sr, s.rhs_jvp(0.0, U, v)) <= 1e-12
    # w / Sr leaves the range of a double for the largest scales: by the exponent that keeps it inside
    e = np.ldexp(1.0, a + 2 * b)
    assert rel_l2(s.rhs_vjp(0.0, U * S, w / Sr * e) * S / e, s.rhs_vjp(0.0, U, w)) <= 1e-12


PROBE = r"""
#include "dg_flux64.cuh"
using namespace apollo;
__device__ unsigned long long ulps(double a, double b) {
  return (unsigned long long)llabs(__double_as_longlong(a) - __double_as_longlong(b));
}
__global__ void k_probe(unsigned long long* worst, int lo, int span, int n) {
  unsigned long long s = 88172645463325252ull + 7919ull * (blockIdx.x * blockDim.x + threadIdx.x), w[3] = {0, 0, 0};
  for (int i = 0; i < n; ++i) {
    s = s * 6364136223846793005ull + 1442695040888963407ull;
    const unsigned long long e = (unsigned long long)(1023 + lo) + (s >> 40) % (unsigned)span;
    const double x = __longlong_as_double((long long)(e << 52 | s >> 12));
    const unsigned long long u[3] = {ulps(recip_normal(x), __drcp_rn(x)), ulps(sqrt_normal(x), __dsqrt_rn(x)),
                                     ulps(rsqrt_normal(x), __drcp_rn(__dsqrt_rn(x)))};
    for (int j = 0; j < 3; ++j) w[j] = u[j] > w[j] ? u[j] : w[j];
  }
  for (int j = 0; j < 3; ++j) atomicMax(worst + j, w[j]);
}
extern "C" int probe(unsigned long long* out, int lo, int span, int n) {
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, 24) != cudaSuccess) return 1;
  cudaMemset(d, 0, 24);
  k_probe<<<296, 256>>>(d, lo, span, n);
  const cudaError_t e = cudaMemcpy(out, d, 24, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e != cudaSuccess;
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("probe")
    (d / "probe.cu").write_text(PROBE)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
                    "-I" + CSRC, "--expt-relaxed-constexpr", "-shared", "-o", str(d / "probe.so"), str(d / "probe.cu")],
                   check=True, capture_output=True)
    return C.CDLL(str(d / "probe.so")).probe


@pytest.mark.parametrize("lo,span", [(-1000, 2000), (-998, 3), (-20, 40), (-402, 4), (398, 4)])
def test_roots(probe, lo, span):
    worst = (C.c_ulonglong * 3)()
    assert probe(worst, lo, span, 2000) == 0
    assert worst[0] <= 1 and worst[1] <= 1 and worst[2] <= 2
