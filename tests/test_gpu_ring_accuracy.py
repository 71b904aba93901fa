"""What the register-resident Jacobi sweep leaves of a sketched split's accuracy:
capped sketches on up to 76 CTAs within 0.2 % of the exact truncation error (the
kept-set stop ends at a tail settled to 1e-3, half of that in the error; the
sketch itself is within 3e-4), and sketches whose rank the cutoff decides."""
import numpy as np
import pytest

import oracle as O
from test_gpu_jacobi_ring import bond

pytestmark = pytest.mark.gpu


def update(engine, sites, gate, cutoff, cap, predicted):
    eng = engine.Engine(mode="chosen", tc_gemm=1)
    p = np.zeros(eng.n_params, dtype=np.float32)
    p[-1] = predicted  # the share of the values that the rank model predicts
    eng.set_rank_params(p, enable=True)
    m = eng.mps(sites, dtype=np.complex64)
    st = m.apply_2q(gate, 1, cutoff, cap)
    a, b = m.site(1), m.site(2)
    m.free()
    eng.close()
    return st, O.theta_of(a.astype(complex), b.astype(complex))


def theta(sites, gate):
    return O.apply_gate_to_theta(O.theta_of(*[t.astype(complex) for t in sites]), gate, sites[0].shape[0],
                                 sites[1].shape[2])


@pytest.mark.parametrize("shape", [(150, 140, 155, 100), (300, 290, 310, 188), (520, 512, 500, 400),
                                   (620, 610, 630, 540)])
def test_capped_sketches_truncate_as_the_exact_split(engine, shape):
    cl, cm, cr, cap = shape
    rng = np.random.default_rng(sum(shape))
    sites = bond(rng, cl, cm, cr, np.exp(-16.0 / cm))
    gate = O.haar_unitary(rng)
    th = theta(sites, gate)
    exact = np.sqrt(np.sum(np.linalg.svd(th, compute_uv=False)[cap:] ** 2))
    st, got = update(engine, sites, gate, 1e-7, cap, 1.0)
    assert st["sketch_size"] > 0 and st["rank"] == cap and not st["fallback"], st
    # FP32 products and sites: some 1e-6 of ||theta||, which exceeds the truncation nowhere here
    assert exact > 1e-4 and np.linalg.norm(got - th) <= 1.002 * exact, (np.linalg.norm(got - th) / exact)


@pytest.mark.parametrize("shape", [(150, 140, 155), (300, 290, 310), (620, 610, 630)])
def test_uncapped_sketches_keep_the_rank_of_the_cutoff(engine, shape):
    cl, cm, cr = shape
    rng = np.random.default_rng(sum(shape))
    sites = bond(rng, cl, cm, cr, np.exp(-40.0 / cm))
    gate = O.haar_unitary(rng)
    th = theta(sites, gate)
    s = np.linalg.svd(th, compute_uv=False)
    tail = np.sqrt(np.cumsum(s[::-1] ** 2))[::-1]
    cutoff = 1e-3
    rank = int(np.sum(tail > cutoff))
    st, got = update(engine, sites, gate, cutoff, 0, 1.25 * rank / len(s) / 1.1)
    assert st["sketch_size"] > rank and not st["fallback"], (st, rank)
    # the rule at the cutoff, one off at a near-tie
    assert abs(st["rank"] - rank) <= 1, (st["rank"], rank)
    kept = st["rank"]
    assert np.linalg.norm(got - th) <= 1.002 * np.sqrt(np.sum(s[kept:] ** 2)) + 1e-5
