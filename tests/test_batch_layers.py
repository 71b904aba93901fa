"""The layers of a batch program may be any iterables of three-part tasks, read
once; what reaches the library is the same, and a task of another length is
refused."""
import ctypes as C
import types

import numpy as np
import pytest


def recording_batch(engine, calls):
    def run(h, p, nlayers, st, circ, site, gates, cutoff, graph):
        def ints(q, n):
            return np.ctypeslib.as_array(C.cast(q, C.POINTER(C.c_int)), (n,)).copy() if n else np.zeros(0, np.int32)
        starts = ints(st, nlayers + 1)
        n = int(starts[-1])
        calls.append((starts, ints(circ, n), ints(site, n),
                      np.ctypeslib.as_array(C.cast(gates, C.POINTER(C.c_double)), (32 * max(n, 1),)).copy()))
        return 0
    b = engine.Batch.__new__(engine.Batch)
    b.eng = types.SimpleNamespace(_lib=types.SimpleNamespace(qt_batch_run=run), _h=None, _check=lambda rc: None)
    b._p, b.ntask = None, 0
    return b


def program():
    rng = np.random.default_rng(1)
    g = [rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4)) for _ in range(5)]
    return [[(0, 1, g[0]), (1, 2, g[1])], [], [(0, 2, g[2]), (1, 1, g[3]), (1, 3, g[4])]]


@pytest.mark.parametrize("kind", ["tuples", "iterators", "generators", "zips", "task iterators", "arrays"])
def test_layers_of_any_iterable(engine, kind):
    layers = program()
    given = {"tuples": lambda l: tuple(l), "iterators": lambda l: iter(l), "generators": lambda l: (t for t in l),
             "zips": lambda l: zip([t[0] for t in l], [t[1] for t in l], [t[2] for t in l]),
             "task iterators": lambda l: [iter(t) for t in l],
             "arrays": lambda l: zip(np.array([t[0] for t in l], int), np.array([t[1] for t in l], int),
                                     [t[2] for t in l])}[kind]
    calls = []
    b = recording_batch(engine, calls)
    b.run(layers, 1e-8)
    b.run([given(l) for l in layers], 1e-8)
    assert b.ntask == 5 and [0, 2, 2, 5] == calls[0][0].tolist()
    assert calls[0][1].tolist() == [0, 1, 0, 1, 1] and calls[0][2].tolist() == [0, 1, 1, 0, 2]
    for x, y in zip(*calls):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("task", [(0, 1), (0, 1, np.eye(4), None)])
def test_tasks_of_another_length_are_refused(engine, task):
    with pytest.raises(ValueError):
        recording_batch(engine, []).run([[task]], 1e-8)
