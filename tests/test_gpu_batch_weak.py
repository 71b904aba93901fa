"""Ensembles of weakly entangling circuits (a disordered Ising chain's evolution)
at a cutoff above the FP32 resolution, with a noise floor above the cutoff: what
no certificate covers is split in FP64, and expectation values are within what
the truncations allow of the statevector's.  (Without that floor the FP32 split
may keep columns that its Jacobi froze, see Batch.run.)"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def ising(rng):
    z, x, one = np.diag([1.0, -1.0]), np.array([[0.0, 1.0], [1.0, 0.0]]), np.eye(2)
    j, hx, hz = rng.uniform(0.5, 1.5, 3)
    h = j * np.kron(z, z) + 0.5 * hx * (np.kron(x, one) + np.kron(one, x)) + 0.25 * hz * (np.kron(z, one) + np.kron(one, z))
    w, v = np.linalg.eigh(h)
    return (v * np.exp(-0.3j * w)) @ v.T


@pytest.mark.parametrize("cutoff", [1e-5, 1e-4])
def test_weakly_entangling_circuits_with_a_noise_floor(engine, cutoff):
    rng = np.random.default_rng(17)
    qubits, depth = [8, 9, 10, 11, 12, 12], [12, 10, 12, 9, 10, 12]
    layers = [[] for _ in range(max(depth))]
    states, updates = [], [0] * len(qubits)
    for c, (n, d) in enumerate(zip(qubits, depth)):
        psi = np.zeros(2 ** n, complex)
        psi[0] = 1
        for layer in range(d):
            for w in range(1 + layer % 2, n, 2):
                g = ising(rng)
                layers[layer].append((c, w, g))
                psi = O.apply_statevector(psi, g, (w, w + 1))
                updates[c] += 1
        states.append(psi)
    eng = engine.Engine(mode="chosen", noise_floor=100 * cutoff)
    b = engine.Batch(eng, qubits, [64] * len(qubits))
    b.run(layers, cutoff)
    assert b.cert_counts()["resolved"] == 0
    for site in (1, 4, 8):
        z = b.expect_z(site)
        for c, (n, psi) in enumerate(zip(qubits, states)):
            # the first site is the fastest bit
            p = (np.abs(psi) ** 2).reshape([2] * n, order="F").sum(tuple(i for i in range(n) if i != site - 1))
            # an update moves the state by the cutoff at most and rounds the two sites it writes to
            # FP32; <Z> of a state of unit norm moves by twice that, its own norm's share once more
            tol = 3 * updates[c] * (cutoff + 2 * 6e-8)
            assert abs(z[c] - (p[0] - p[1])) <= tol, (c, site, z[c], p[0] - p[1], tol)
    b.free()
    eng.close()
