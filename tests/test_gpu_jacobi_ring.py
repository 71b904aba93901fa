"""The register-resident FP32 Jacobi sweep, which splits the sketch of a capped
update: sketches on odd, even and power-of-two numbers of CTAs, one to sixteen
warps with two and four rows per lane and ragged last slices, against the exact
split and against the Gram-based sweep kernel; its results do not vary between
runs, and a wait that nothing ends returns an error."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def sketching_engine(engine):
    eng = engine.Engine(mode="chosen", tc_gemm=1)
    p = np.zeros(eng.n_params, dtype=np.float32)
    p[-1] = 1.0  # a rank model predicting the cap: the update is sketched
    eng.set_rank_params(p, enable=True)
    return eng


def bond(rng, cl, cm, cr, decay):
    def iso(rows, cols):
        return np.linalg.qr(rng.standard_normal((rows, cols)) + 1j * rng.standard_normal((rows, cols)))[0]
    s = decay ** np.arange(cm)
    a = iso(max(2 * cl, cm), cm)[:2 * cl] * (s / np.linalg.norm(s))
    b = iso(max(2 * cr, cm), cm)[:2 * cr].conj().T
    return [a.reshape((cl, 2, cm), order="F").astype(np.complex64),
            b.reshape((cm, 2, cr), order="F").astype(np.complex64)]


# chiL, chiM, chiR, cap: sketches of cap + 64 (or 1.125 cap) columns, 8 per CTA
@pytest.mark.parametrize("shape", [(90, 90, 95, 50), (130, 128, 127, 96), (150, 140, 155, 100), (257, 250, 260, 130),
                                   (300, 290, 310, 188), (520, 512, 500, 400), (700, 690, 1000, 448)])
def test_ring_splits_sketches(engine, monkeypatch, shape):
    cl, cm, cr, cap = shape
    rng = np.random.default_rng(sum(shape))
    sites = bond(rng, cl, cm, cr, np.exp(-26.0 / cm))
    g = O.haar_unitary(rng)
    th = O.apply_gate_to_theta(O.theta_of(*[t.astype(complex) for t in sites]), g, cl, cr)
    ref = np.linalg.svd(th, compute_uv=False)
    exact = np.sqrt(np.sum(ref[cap:] ** 2))
    for ring in ("1", "0"):
        monkeypatch.setenv("QT_JACOBI_RING", ring)
        first = None
        for _ in range(2):
            eng = sketching_engine(engine)
            m = eng.mps(sites, dtype=np.complex64)
            st = m.apply_2q(g, 1, 1e-7, cap)
            a, b = m.site(1), m.site(2)
            m.free()
            eng.close()
            assert st["sketch_size"] > 0 and st["rank"] == cap and not st["fallback"], st
            # the bounds of the other capped sketches: 1.1x the exact truncation error (plus
            # FP32 rounding), a left factor orthonormal to rounding
            assert np.linalg.norm(th - O.theta_of(a.astype(complex), b.astype(complex))) <= 1.1 * exact + 1e-5
            u = a.reshape((2 * cl, cap), order="F").astype(complex)
            assert np.abs(u.conj().T @ u - np.eye(cap)).max() <= 2e-6 * np.sqrt(2 * cl)
            if first is not None:
                assert np.array_equal(first[0], a) and np.array_equal(first[1], b)
            first = (a, b)


def test_ring_wait_times_out_and_the_handle_recovers(engine, monkeypatch):
    rng = np.random.default_rng(3)
    sites = bond(rng, 150, 140, 155, np.exp(-26.0 / 140))
    g = O.haar_unitary(rng)
    eng = sketching_engine(engine)
    m = eng.mps(sites, dtype=np.complex64)
    monkeypatch.setenv("QT_JACOBI_STALL_TEST", "20000")
    with pytest.raises(engine.EngineError) as e:
        m.apply_2q(g, 1, 1e-7, 100)
    assert e.value.code == engine.QT_ETIMEOUT
    m.free()
    monkeypatch.delenv("QT_JACOBI_STALL_TEST")
    m = eng.mps(sites, dtype=np.complex64)
    st = m.apply_2q(g, 1, 1e-7, 100)
    assert st["rank"] == 100 and st["sketch_size"] > 0 and not st["fallback"], st
    m.free()
    eng.close()
