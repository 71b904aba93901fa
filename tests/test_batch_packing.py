"""Packing of a batch program's gates: each gate's entries column-major as
interleaved doubles, whatever the gates' shapes, types and strides."""
import numpy as np
import pytest


def one_by_one(gates):
    flat = [np.asarray(g, dtype=np.complex128).reshape(-1, order="F") for g in gates]
    return np.concatenate([np.stack([f.real, f.imag], axis=1).ravel() for f in flat])


@pytest.mark.parametrize("kind", ["square", "legs", "flat", "lists", "real", "single", "views", "mixed"])
def test_packed_gates_match_one_by_one(engine, kind):
    rng = np.random.default_rng(0)
    g = [rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4)) for _ in range(5)]
    gates = {"square": g, "legs": [x.reshape((2, 2, 2, 2), order="F") for x in g], "flat": [x.reshape(-1) for x in g],
             "lists": [x.tolist() for x in g], "real": [x.real for x in g], "single": [x.astype(np.complex64) for x in g],
             "views": [x.T[::-1] for x in g], "mixed": [g[0], g[1].reshape((2, 2, 2, 2), order="F"), g[2].tolist()]}[kind]
    got = engine.Batch._pack_gates(gates)
    assert got.dtype == np.float64 and got.flags["C_CONTIGUOUS"] and np.array_equal(got, one_by_one(gates))
    assert engine.Batch._pack_gates([]).size == 32
