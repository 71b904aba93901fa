"""The rotation of a column pair in unevaluated FP32 pairs (cta_angle) against its
FP64 evaluation (cta_angle64), on the device and bit for bit: the same decision,
cosine, sine and phase, over random sums and the places where the two could part
-- nearly equal norms, norms 1e15 apart, phases with a tiny component, cosines at
the tolerance and at 1, the ends of the range that stays in FP32, zeros,
denormals, infinities and NaN."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qaintensor.jl_gb300")

SOURCE = r"""
#include "qt_cta.cuh"
__global__ void both(int n, const float* x, double tol, double nu2, float* y) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float* a = x + 4 * (size_t)i;
    const cta_rotation<float> p = cta_angle(a[0], a[1], a[2], a[3], tol, (float)(tol * tol), nu2, __double2float_rd(nu2));
    const cta_rotation<float> q = cta_angle64<float>(a[0], a[1], a[2], a[3], tol, nu2);
    float* o = y + 10 * (size_t)i;
    o[0] = p.c; o[1] = p.s; o[2] = p.er; o[3] = p.ei; o[4] = p.on;
    o[5] = q.c; o[6] = q.s; o[7] = q.er; o[8] = q.ei; o[9] = q.on;
  }
}
extern "C" int angles(int n, const float* x, double tol, double nu2, float* y) {
  float *dx = nullptr, *dy = nullptr;
  cudaError_t e = cudaMalloc(&dx, sizeof(float) * 4 * (size_t)n);
  if (e == cudaSuccess) e = cudaMalloc(&dy, sizeof(float) * 10 * (size_t)n);
  if (e == cudaSuccess) e = cudaMemcpy(dx, x, sizeof(float) * 4 * (size_t)n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) { both<<<608, 256>>>(n, dx, tol, nu2, dy); e = cudaGetLastError(); }
  if (e == cudaSuccess) e = cudaMemcpy(y, dy, sizeof(float) * 10 * (size_t)n, cudaMemcpyDeviceToHost);
  cudaFree(dx);
  cudaFree(dy);
  return (int)e;
}
"""


@pytest.fixture(scope="module")
def angles(tmp_path_factory):
    sys.path.insert(0, PKG)
    try:
        import build  # the engine's compiler and flags
    finally:
        sys.path.pop(0)
    d = tmp_path_factory.mktemp("angle")
    src, lib = str(d / "angle.cu"), str(d / "libangle.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    r = subprocess.run([build.nvcc(), *build.ARCH, *build.FLAGS, "-shared", "-o", lib, src], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    f = C.CDLL(lib).angles
    f.argtypes = [C.c_int, C.c_void_p, C.c_double, C.c_double, C.c_void_p]

    def run(x, tol, nu2):
        x = np.ascontiguousarray(x, np.float32)
        y = np.empty((len(x), 10), np.float32)
        assert f(len(x), x.ctypes.data, tol, nu2, y.ctypes.data) == 0
        return y[:, :5], y[:, 5:]
    return run


def sums(rng, kind, n, tol):
    """(aa, bb, gr, gi) of n pairs."""
    log = lambda lo, hi: 10.0 ** rng.uniform(lo, hi, n)  # noqa: E731
    aa = log(-3, 3)
    bb = aa * log(-2, 2)
    cos, phi = rng.uniform(0, 1, n), rng.uniform(-np.pi, np.pi, n)
    if kind == "equal":  # norms a few units in the last place apart, or the same
        bb = aa.astype(np.float32) * (1 + rng.integers(-8, 9, n) * 2.0 ** -23)
        cos = log(-7, 0)
    elif kind == "apart":
        bb = aa * log(-15, 15)
        cos = log(-7, 0)
    elif kind == "phase":
        phi = rng.integers(0, 4, n) * np.pi / 2 + rng.choice([-1, 1], n) * log(-40, -1)
    elif kind == "tolerance":
        cos = tol * (1 + rng.choice([-1, 1], n) * log(-8, -3))
    elif kind == "aligned":
        cos = 1 - log(-8, -1)
    elif kind == "range":
        aa, bb = log(-31, -29), log(-31, -29)
        up = rng.random(n) < 0.5
        aa, bb = np.where(up, aa * 1e60, aa), np.where(up, bb * 1e60, bb)
        cos = log(-7, 0)
    elif kind == "steep":  # zeta = (bb - aa) / 2 |gamma| around 1e15
        bb = aa * log(14, 17)
        cos = log(-8, 0)
    g = cos * np.sqrt(aa * bb)
    with np.errstate(over="ignore", under="ignore"):
        return np.stack([aa, bb, g * np.cos(phi), g * np.sin(phi)], 1).astype(np.float32)


KINDS = ["random", "equal", "apart", "phase", "tolerance", "aligned", "range", "steep"]


@pytest.mark.parametrize("tol", [16 * 5.96e-8, 1e-4])
@pytest.mark.parametrize("kind", KINDS + ["special"])
def test_same_bits_as_in_fp64(angles, kind, tol):
    rng = np.random.default_rng(len(kind))
    if kind == "special":
        v = np.array([0, -0.0, 1, -1, 1e-45, -1e-40, 1.2e-38, 7.8e-31, 7.9e-31, 8e-31, 1e-15, 1e15, 1.19e30, 1.2e30,
                      1.21e30, 3e38, np.inf, -np.inf, np.nan], np.float32)
        x = np.stack([a.ravel() for a in np.meshgrid(np.abs(v), np.abs(v), v, v)], 1)
    else:
        x = sums(rng, kind, 4_000_000, tol)
    for nu2 in (0.0, 1e-12, 0.3):
        got, want = angles(x, tol, nu2)
        same = (got.view(np.int32) == want.view(np.int32)).all(1)
        # (a rotation of NaN is not taken; infinite sums that pass the test give NaN in both)
        same |= (np.isnan(got) == np.isnan(want)).all(1) & np.isnan(want).any(1)
        bad = np.nonzero(~same)[0]
        assert len(bad) == 0, (len(bad), x[bad[:5]], got[bad[:5]], want[bad[:5]])
        if kind not in ("special", "range") and nu2 == 0.0:
            assert want[:, 4].any()
