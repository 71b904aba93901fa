"""The batched layer kernel over its launch shapes and theta' sizes: rows per
lane 1, 2, 4 and 8, theta' in shared memory and above it, wide and tall,
odd bond caps, against the dense statevector (no truncation: every cap holds
the circuit's full rank) and against the FP64 oracle (caps that truncate)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def run_circuits(engine, circuits, cutoff, shape):
    eng = engine.Engine(mode="chosen")
    b = engine.Batch(eng, [c[0] for c in circuits], [c[2] for c in circuits])
    for bucket in (16, 32, 64, 128):
        b.set_launch(bucket, *shape)
    layers = [[] for _ in range(max(c[1] for c in circuits))]
    for ci, (_, _, _, gates) in enumerate(circuits):
        for (layer, w, g) in gates:
            layers[layer - 1].append((ci, w, g))
    b.run(layers, cutoff)
    psi = [O.mps_to_state([b.site(ci, i).astype(np.complex128) for i in range(1, c[0] + 1)])
           for ci, c in enumerate(circuits)]
    z = [b.expect_z(w) for w in range(1, min(c[0] for c in circuits) + 1)]
    dims = [list(b.bond_dims(ci)) for ci in range(len(circuits))]
    b.free()
    eng.close()
    return psi, z, dims


@pytest.mark.parametrize("shape", [(128, 4), (256, 1), (512, 2), (1024, 1)])
def test_full_rank_circuits_match_the_statevector(engine, shape):
    rng = np.random.default_rng(77)
    circuits = []
    for n, cap in [(2, 1), (2, 3), (5, 7), (8, 16), (9, 17), (10, 32), (11, 33), (12, 64), (13, 65), (15, 128)]:
        depth = 4 if cap < 4 else 2 * n // 3
        circuits.append((n, depth, cap if n > 2 else 2, O.brickwork_gates(n, depth, rng)))
    psi, z, dims = run_circuits(engine, circuits, 1e-8, shape)
    for ci, (n, depth, cap, gates) in enumerate(circuits):
        dense = np.zeros(2 ** n, dtype=complex)
        dense[0] = 1
        for (_, w, g) in gates:
            dense = O.apply_statevector(dense, g, (w, w + 1))
        # FP32 storage and arithmetic: 5e-5 over 6 layers, in proportion to the depth
        assert np.linalg.norm(psi[ci] - dense) <= 5e-5 * max(1.0, depth / 6), (n, cap)
        for w in range(2):
            p = np.abs(dense.reshape((2,) * n, order="F")) ** 2
            p0, p1 = p.take(0, axis=w).sum(), p.take(1, axis=w).sum()
            assert abs(z[w][ci] - (p0 - p1) / (p0 + p1)) <= 1e-4 * max(1.0, depth / 6), (n, cap, w)


def test_truncating_caps_match_the_oracle(engine):
    # gates near the identity: spectra that fall fast, so that the caps cut
    # where the kept space is well defined
    rng = np.random.default_rng(78)
    circuits = []
    for n, cap in [(7, 3), (9, 5), (10, 15), (12, 20)]:
        gates = []
        for (layer, w, _) in O.brickwork_gates(n, 10, rng):
            a = rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4))
            lam, v = np.linalg.eigh(a + a.conj().T)
            gates.append((layer, w, (v * np.exp(-0.15j * lam)) @ v.conj().T))
        circuits.append((n, 10, cap, gates))
    cutoff = 1e-5  # above the FP32 resolution: the rule decides as in FP64 up to near-ties
    psi, z, dims = run_circuits(engine, circuits, cutoff, (256, 1))
    for ci, (n, depth, cap, gates) in enumerate(circuits):
        sites, _ = O.run_brickwork(n, gates, cutoff, cap)
        ref = O.mps_to_state(sites)
        assert max(dims[ci]) <= cap
        # FP32 errors as above, plus a value dropped on one side of the cutoff only, at most once per update
        bound = (5e-5 * depth / 6 + cutoff * np.sqrt(len(gates))) * np.linalg.norm(ref)
        assert np.linalg.norm(psi[ci] - ref) <= bound, (n, cap)
