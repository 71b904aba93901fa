"""A two-site update beside a bond of more columns than the second dimension of a
grid takes in tiles of eight (65535 x 8 = 524280): an end of a chain whose third
tensor is that long, in FP64 products of both element types."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chir", [524280, 524281, 600001])
@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
def test_update_beside_a_long_bond(engine, chir, dtype):
    rng = np.random.default_rng(chir)

    def unit(*shape):
        x = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
        return np.asfortranarray((x / np.linalg.norm(x)).astype(dtype))

    sites = [unit(1, 2, 2), unit(2, 2, chir), unit(chir, 2, 1)]
    gate = O.haar_unitary(rng)
    theta = np.einsum("pqrs,arsb->apqb", gate.reshape((2, 2, 2, 2), order="F"),
                      np.tensordot(sites[0].astype(complex), sites[1].astype(complex), 1))
    eng = engine.Engine(mode="plain")
    mps = eng.mps(sites, dtype=dtype)
    st = mps.apply_2q(gate, 1, 0.0, 0)
    assert st["rank"] == 2
    got = np.tensordot(mps.site(1).astype(complex), mps.site(2).astype(complex), 1)
    # FP64 throughout; complex64 rounds the two tensors as it stores them
    tol = 1e-12 if dtype == np.complex128 else 4 * 6e-8
    assert np.linalg.norm(got - theta) <= tol * np.linalg.norm(theta)
    mps.free()
    eng.close()
