"""The FP64 cluster round at the edges of its shapes: one to eight CTAs per
pair, row slices with and without remainder, V beside X and after it, column
counts off the 8-column block, norms far from 1, spectra over 14 decades and
equal singular values, against LAPACK."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def crandn(rng, *shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) / np.sqrt(2)


def with_spectrum(rng, m, n, s):
    k = min(m, n)
    q1, _ = np.linalg.qr(crandn(rng, m, k))
    q2, _ = np.linalg.qr(crandn(rng, n, k))
    return (q1 * s) @ q2.conj().T


@pytest.mark.parametrize("cluster", ["", "1", "2", "4", "8"])
@pytest.mark.parametrize("shape", [(2, 2), (9, 7), (17, 16), (33, 31), (64, 64), (65, 129), (130, 127), (257, 40)])
def test_fp64_round_shapes(engine, monkeypatch, shape, cluster):
    if cluster:
        monkeypatch.setenv("QT_JACOBI_CLUSTER", cluster)
    m, n = shape
    rng = np.random.default_rng(m * 1000 + n)
    k = min(m, n)
    for s, scale in [(0.9 ** np.arange(k), 1.0), (10.0 ** (-14.0 * np.arange(k) / k), 1e90), (np.ones(k), 1e-90),
                     (np.repeat(1.0 + 1e-9 * np.arange((k + 1) // 2), 2)[:k][::-1].copy(), 3.0)]:
        M = with_spectrum(rng, m, n, s) * scale
        eng = engine.Engine(mode="plain")
        U, S, Vh, kk, _ = eng.truncated_svd(M, 0.0)
        eng.close()
        ref = np.linalg.svd(M, compute_uv=False)
        # backward error of a product of unitary transformations: a small
        # multiple of u per sweep and entry, 1e-12 as for the other rounds
        assert kk == k
        assert np.abs(S - ref).max() <= 1e-12 * ref[0]
        assert np.linalg.norm((U * S) @ Vh - M) <= 1e-12 * np.sqrt(max(m, n)) * np.linalg.norm(M)
        assert np.abs(U.conj().T @ U - np.eye(k)).max() <= 1e-11
