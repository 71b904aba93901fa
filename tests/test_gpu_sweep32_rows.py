"""The FP32 sweep kernel where V's rows ride beside X's: X ending inside a
warp's 32 rows, at and just past a slab of 256, V's rows in the idle warps,
behind X's, or both, and matrices split over two CTAs per pair."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(16, 16), (31, 33), (33, 97), (97, 31), (96, 160), (160, 97), (224, 33), (225, 225),
                                   (256, 41), (257, 40), (130, 290), (512, 24), (513, 289), (601, 530)])
def test_fp32_split_at_row_edges(engine, shape):
    m, n = shape
    rng = np.random.default_rng(3 * m + n)
    k0 = min(m, n)
    q1, _ = np.linalg.qr(rng.standard_normal((m, k0)) + 1j * rng.standard_normal((m, k0)))
    q2, _ = np.linalg.qr(rng.standard_normal((n, k0)) + 1j * rng.standard_normal((n, k0)))
    M = ((q1 * 0.9 ** np.arange(k0)) @ q2.conj().T).astype(np.complex64)
    ref = np.linalg.svd(M.astype(np.complex128), compute_uv=False)
    # the FP32 resolution, and a cutoff well above it
    floor = 4 * np.sqrt(max(m, n)) * 5.96e-8 * np.linalg.norm(ref)
    cut = 50 * floor
    eng = engine.Engine(mode="chosen", jacobi_kernel=0)
    U, S, Vh, k, _ = eng.truncated_svd(M, cut, mode="chosen")
    eng.close()
    tail = np.sqrt(np.cumsum(ref[::-1] ** 2))[::-1]
    assert abs(k - (int(np.argmax(np.append(tail[1:], 0.0) <= cut)) + 1)) <= 1
    assert np.abs(S[:k] - ref[:k]).max() <= 2 * floor
    assert np.linalg.norm((U * S) @ Vh - M) <= 1.1 * np.sqrt(np.sum(ref[k:] ** 2)) + floor
    assert np.abs(U.conj().T @ U - np.eye(k)).max() <= 2e-6 * np.sqrt(m)
