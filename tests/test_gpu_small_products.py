"""FP64 and FP32 products whose tile is chosen by the grid they give (16, 32 and
64 wide), over remainders of each tile and both operand forms, and the FP64
orthonormalisation through MPS compression, at block and chunk remainders."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def crandn(rng, *shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) / np.sqrt(2)


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("shape", [(1, 1, 1), (15, 17, 33), (16, 16, 16), (64, 64, 5), (65, 31, 200), (300, 500, 40),
                                   (560, 560, 17), (577, 1100, 9)])
def test_products_match_numpy(engine, shape, dtype):
    m, n, k = shape
    rng = np.random.default_rng(m + 10 * n + 100 * k)
    eng = engine.Engine(mode="plain")
    for op_a in "NC":
        for op_b in "NC":
            a = crandn(rng, *((m, k) if op_a == "N" else (k, m))).astype(dtype)
            b = crandn(rng, *((k, n) if op_b == "N" else (n, k))).astype(dtype)
            c = crandn(rng, m, n).astype(dtype)
            got = eng.gemm(a, b, op_a, op_b, alpha=0.5 - 2j, beta=1.5j, out=c)
            x = a if op_a == "N" else a.conj().T
            y = b if op_b == "N" else b.conj().T
            ref = (0.5 - 2j) * (x.astype(complex) @ y.astype(complex)) + 1.5j * c
            u = 1.11e-16 if dtype == np.complex128 else 5.96e-8
            # k + 3 roundings of u each on sums of k terms of size ~1 (a few u of slack each)
            assert np.abs(got - ref).max() <= 8 * (k + 3) * u * max(1.0, np.abs(ref).max())
    eng.close()


@pytest.mark.parametrize("chi", [1, 7, 31, 32, 33, 70])
def test_fp64_left_canonical_sites_are_isometries(engine, chi):
    rng = np.random.default_rng(chi)
    n = 6
    dims = [1] + [chi] * (n - 1) + [1]
    # column norms over twelve decades: blocks of condition 1e12
    sites = [crandn(rng, dims[i], 2, dims[i + 1]) * 10.0 ** (-12.0 * np.arange(dims[i + 1]) / dims[i + 1])
             for i in range(n)]
    eng = engine.Engine(mode="plain")
    mps = eng.mps(sites, dtype=np.complex128)
    before = mps.norm2()
    mps.compress(0.0, 0, mode="plain", normalize=False)
    # right-canonical after the compression: every site but the first an isometry
    for i in range(2, n + 1):
        t = mps.site(i)
        g = np.tensordot(t, t.conj(), ([1, 2], [1, 2]))
        assert np.abs(g - np.eye(t.shape[0])).max() <= 1e-11
    assert abs(mps.norm2() - before) <= 1e-11 * before
    mps.free()
    eng.close()
