"""Expectation values through both environments: chains of one and two sites, the
measured site at either end, open boundary legs, ragged tiles and both element
types against numpy, and an environment of more than 2^31 entries."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chain(rng, dims, dtype):
    return [np.asfortranarray((rng.standard_normal((dims[i], 2, dims[i + 1])) +
                               1j * rng.standard_normal((dims[i], 2, dims[i + 1]))).astype(dtype)
                              / np.sqrt(4 * dims[i])) for i in range(len(dims) - 1)]


def expect(sites, ops):
    env = np.eye(sites[0].shape[0], dtype=complex)
    for i, a in enumerate(np.asarray(s, complex) for s in sites):
        b = a * np.array([1.0, -1.0])[None, :, None] if i in ops else a
        env = np.tensordot(a.conj(), np.tensordot(env, b, 1), ([0, 1], [0, 1]))
    return np.trace(env).real


# bond dimensions of the chains; the outer ones are traced
@pytest.mark.parametrize("dims", [(1, 1), (3, 5), (17, 16), (1, 2, 1), (2, 33, 3), (1, 2, 4, 2, 1), (5, 15, 16, 17, 7),
                                  (1, 31, 47, 65, 130, 9), (40, 3, 1, 20, 70)])
@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
def test_expectation_values_of_ragged_and_open_chains(engine, dims, dtype):
    sites = chain(np.random.default_rng(sum(dims)), dims, dtype)
    n = len(sites)
    eng = engine.Engine(mode="plain")
    mps = eng.mps(sites, dtype=dtype)
    sites = [mps.site(i + 1) for i in range(n)]  # as stored
    norm2 = expect(sites, ())
    # FP64 sums of positive squares: some 1e-16 per product and site
    tol = 1e-12
    assert abs(mps.norm2() - norm2) <= tol * norm2
    for i in range(n):
        assert abs(mps.expect_z(i + 1) - expect(sites, (i,)) / norm2) <= tol
    for i in range(n - 1):
        assert abs(mps.expect_zz(i + 1) - expect(sites, (i, i + 1)) / norm2) <= tol
    mps.free()
    eng.close()


def test_environment_of_more_than_2_31_entries(engine):
    chi = 46342  # 34 GB an environment, three of them
    free, total = ctypes.c_size_t(), ctypes.c_size_t()
    eng = engine.Engine(mode="plain")
    rt = ctypes.CDLL("libcudart.so.13")
    if rt.cudaMemGetInfo(ctypes.byref(free), ctypes.byref(total)) != 0 or free.value < 150e9:
        eng.close()
        pytest.skip("needs 150 GB of free device memory")
    sites = chain(np.random.default_rng(1), (1, chi, 1), np.complex64)
    mps = eng.mps(sites, dtype=np.complex64)
    pair = np.tensordot(*[mps.site(i).astype(complex) for i in (1, 2)], 1)[0, :, :, 0]
    p = np.abs(pair) ** 2
    assert abs(mps.expect_z(1) - (p[0].sum() - p[1].sum()) / p.sum()) <= 1e-10
    mps.free()
    eng.close()
