"""Updates under a small sweep limit: FP64 splits of small bonds and sketched FP32
splits are done within as few sweeps as the rounds that need the fewest take."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def bond(rng, cl, cm, cr, decay):
    def iso(rows, cols):
        return np.linalg.qr(rng.standard_normal((rows, cols)) + 1j * rng.standard_normal((rows, cols)))[0]
    s = decay ** np.arange(cm)
    a = iso(max(2 * cl, cm), cm)[:2 * cl] * (s / np.linalg.norm(s))
    b = iso(max(2 * cr, cm), cm)[:2 * cr].conj().T
    return [a.reshape((cl, 2, cm), order="F"), b.reshape((cm, 2, cr), order="F")]


def update(engine, sites, gate, limit, cutoff, cap, **cfg):
    eng = engine.Engine(max_sweeps=limit, **cfg)
    if cap:
        p = np.zeros(eng.n_params, dtype=np.float32)
        p[-1] = 1.0  # a rank model predicting the cap: the update is sketched
        eng.set_rank_params(p, enable=True)
    m = eng.mps(sites, dtype=sites[0].dtype)
    st = m.apply_2q(gate, 1, cutoff, cap)
    a, b = m.site(1), m.site(2)
    m.free()
    eng.close()
    return st, a, b


# bond and the sweeps that FP64 pair solves to the end need
@pytest.mark.parametrize("case", [(2, 2), (3, 2), (4, 2), (6, 2), (8, 2), (12, 5), (16, 5), (24, 6), (32, 7), (64, 8)])
@pytest.mark.parametrize("decay", [1.0, 0.5])
def test_fp64_splits_under_a_small_limit(engine, case, decay):
    chi, limit = case
    rng = np.random.default_rng(chi)
    sites = bond(rng, chi, chi, chi, decay)
    gate = O.haar_unitary(rng)
    th = O.apply_gate_to_theta(O.theta_of(*sites), gate, chi, chi)
    st, a, b = update(engine, sites, gate, limit, 1e-10, 0, mode="plain")
    assert st["sweeps"] <= limit
    # every value is kept but those below 1e-10: FP64 products, at any state of the Jacobi
    assert np.linalg.norm(th - O.theta_of(a, b)) <= 1e-9
    u = a.reshape((2 * chi, -1), order="F")
    assert np.abs(u.conj().T @ u - np.eye(u.shape[1])).max() <= 1e-11


@pytest.mark.parametrize("case", [(90, 90, 95, 50, 4), (150, 140, 155, 100, 4), (300, 290, 310, 188, 4),
                                  (520, 512, 500, 400, 5)])
def test_sketched_splits_under_a_small_limit(engine, case):
    cl, cm, cr, cap, limit = case
    rng = np.random.default_rng(cl)
    sites = [t.astype(np.complex64) for t in bond(rng, cl, cm, cr, np.exp(-26.0 / cm))]
    gate = O.haar_unitary(rng)
    th = O.apply_gate_to_theta(O.theta_of(*[t.astype(complex) for t in sites]), gate, cl, cr)
    exact = np.sqrt(np.sum(np.linalg.svd(th, compute_uv=False)[cap:] ** 2))
    st, a, b = update(engine, sites, gate, limit, 1e-7, cap, mode="chosen", tc_gemm=1)
    assert st["sketch_size"] > 0 and st["rank"] == cap and not st["fallback"], st
    # the bounds of the other capped sketches
    assert np.linalg.norm(th - O.theta_of(a.astype(complex), b.astype(complex))) <= 1.1 * exact + 1e-5
