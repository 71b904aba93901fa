"""FP64 splits of a layer that leaves many tasks: one CTA a task instead of a
cluster.  A circuit comes out the same, bit for bit, alone and among enough
copies of itself, in every bucket of caps, with the columns in shared memory
and in the slab; and a layer of as many tasks as fit on the chip takes about as
long as a layer of few.  A noise floor above ||theta'|| leaves every task to
the FP64 split."""
import time

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def run(engine, n, cap, depth, copies):
    """The program's batch: `copies` of one circuit."""
    gates = O.brickwork_gates(n, depth, np.random.default_rng(n * cap))
    eng = engine.Engine(mode="chosen", noise_floor=10.0)
    b = engine.Batch(eng, [n] * copies, [cap] * copies)
    layers = [[] for _ in range(depth)]
    for (layer, w, g) in gates:
        layers[layer - 1] += [(c, w, g) for c in range(copies)]
    b.run(layers, 1e-12)
    assert b.cert_counts()["fallback"] == len(gates) * copies
    return eng, b


# tasks of a layer: (n - 1) / 2 a copy; copies above and below the lines of 28, 76, 100 and 300 tasks
@pytest.mark.parametrize("case", [(2, 2, 2, 40), (5, 5, 5, 20), (7, 9, 7, 12), (8, 16, 8, 12), (9, 17, 8, 24),
                                  (10, 32, 9, 20), (12, 64, 10, 22), (13, 50, 8, 20), (14, 128, 9, 48)])
def test_alone_and_cluster_splits_give_the_same_bits(engine, case):
    n, cap, depth, copies = case
    eng, b = run(engine, n, cap, depth, 1)
    want = [b.site(0, i) for i in range(1, n + 1)]
    stats = b.task_stats()
    b.free()
    eng.close()
    eng, b = run(engine, n, cap, depth, copies)
    for c in (0, copies // 2, copies - 1):
        for i in range(1, n + 1):
            assert np.array_equal(want[i - 1], b.site(c, i)), (c, i)
    for one, many in zip(stats, b.task_stats()):
        # every layer lists each task `copies` times in a row
        assert np.array_equal(np.repeat(one, copies), many)
    b.free()
    eng.close()


def test_a_layer_of_many_tasks_takes_as_long_as_one_of_few(engine):
    best = {}
    for copies in (8, 64):  # 24 and 192 tasks a layer on 152 SMs: one turn and two
        eng, b = run(engine, 6, 8, 6, copies)
        best[copies] = 1e9
        for _ in range(8):
            b.reset()
            t = time.perf_counter()
            b.replay()
            best[copies] = min(best[copies], time.perf_counter() - t)
        b.free()
        eng.close()
    assert best[64] <= 3 * best[8], best
