"""The batched layer's FP64 split (a cluster of CTAs per task, rows split over
them) over its slice heights: up to 8, 16 and 32 rows per CTA, ragged slices,
fewer rows than CTAs, wide and tall, against the dense statevector.  A noise
floor above ||theta'|| leaves no decision to the FP32 split, so that every
task takes the FP64 one."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("circuits", [[(2, 2), (3, 2), (4, 4), (5, 5), (7, 9)], [(8, 16), (9, 17), (10, 32), (11, 33)],
                                      [(12, 64), (13, 65), (15, 128)]])
def test_fp64_split_matches_the_statevector(engine, circuits):
    rng = np.random.default_rng(91)
    eng = engine.Engine(mode="chosen", noise_floor=10.0)
    b = engine.Batch(eng, [n for n, _ in circuits], [cap for _, cap in circuits])
    gates = [O.brickwork_gates(n, n - 1, rng) for n, _ in circuits]
    layers = [[] for _ in range(max(n - 1 for n, _ in circuits))]
    for ci, gs in enumerate(gates):
        for (layer, w, g) in gs:
            layers[layer - 1].append((ci, w, g))
    b.run(layers, 1e-12)
    cert = b.cert_counts()
    assert cert["fallback"] == sum(map(len, layers)), cert
    for ci, (n, cap) in enumerate(circuits):
        dims = [int(d) for d in b.bond_dims(ci)]
        assert max(dims) >= 2 ** (n // 2), (n, dims)
        dense = np.zeros(2 ** n, dtype=complex)
        dense[0] = 1
        for (_, w, g) in gates[ci]:
            dense = O.apply_statevector(dense, g, (w, w + 1))
        psi = O.mps_to_state([b.site(ci, i).astype(np.complex128) for i in range(1, n + 1)])
        # FP64 but for the sites: each update rounds the two it writes to FP32, 2 x 6e-8 of the state at most
        assert np.linalg.norm(psi - dense) <= 1.2e-7 * len(gates[ci]), (n, dims)
    # the captured program again, from |0...0>: the same splits
    ranks = b.task_stats()[0].copy()
    b.reset()
    b.replay()
    assert np.array_equal(ranks, b.task_stats()[0])
    b.free()
    eng.close()
