"""qt_jacobi_svd on FP32 storage refuses a matrix that holds a NaN or an infinity,
with pairwise rotations (the register-resident sweep) and without; the caller's
handle computes normally afterwards."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def jacobi(engine, eng, M, pairwise):
    torch = pytest.importorskip("torch")
    f = engine.library()._Z13qt_jacobi_svdI6float2EiP9qt_handlePT_lllS4_ldiPidib
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int64, C.c_int64, C.c_int64, C.c_void_p, C.c_int64, C.c_double, C.c_int,
                  C.POINTER(C.c_int), C.c_double, C.c_int, C.c_bool]
    m, n = M.shape
    X = torch.from_numpy(np.ascontiguousarray(M.T)).cuda()  # column-major
    torch.cuda.synchronize()
    sweeps = C.c_int()
    rc = f(eng._h, X.data_ptr(), m, n, m, None, n, 1e-6, 40, C.byref(sweeps), -1.0, 0, pairwise)
    assert eng._lib.qt_sync(eng._h) == 0
    return rc, X.cpu().numpy().T


@pytest.mark.parametrize("pairwise", [True, False])
@pytest.mark.parametrize("shape", [(40, 24), (200, 64), (700, 130)])
def test_nonfinite_columns_are_refused(engine, shape, pairwise):
    rng = np.random.default_rng(sum(shape))
    M = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
    eng = engine.Engine(mode="chosen")
    for value in (np.nan, np.inf, complex(0, -np.inf)):
        for (i, j) in ((0, 0), (shape[0] - 1, shape[1] // 2), (shape[0] // 2, shape[1] - 1)):
            bad = M.copy()
            bad[i, j] = value
            assert jacobi(engine, eng, bad, pairwise)[0] == engine.QT_ENUMERIC
    rc, X = jacobi(engine, eng, M, pairwise)
    G = X.conj().T.astype(complex) @ X.astype(complex)
    d = np.sqrt(np.diag(G).real)
    # the columns' cosines, to the tolerance asked for and FP32 sums of `rows` products
    off = np.abs((G - np.diag(d ** 2)) / np.outer(d, d)).max()
    assert rc == 0 and off <= 1e-6 + 4 * np.sqrt(shape[0]) * 6e-8, (rc, off)
    eng.close()
