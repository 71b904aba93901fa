"""Work that users of the framework have it do, as cases for timing and comparison.

A case is a dict of plain values.  ``listed()`` gives a dozen of them,
``draw(rng)`` further ones of the same ranges, ``prepare(case, seed)`` what a
program holds before the call, ``run(state)`` one pass through the public
entry points, ``work(case)`` the bytes and flops that pass cannot do without
and ``exact(case, seed)`` its outputs as numpy computes them in 64 bits.

Outputs are the quantities that a split leaves well defined: a site tensor is
fixed only up to a unitary on its bonds, so an updated pair is returned as its
two-site tensor and a chain of few sites as its amplitudes.  Ensembles and
long chains return the expectation values that such programs are run for.

Kinds of case:
  bond     one two-qubit gate (or leg swap) and split on a bond held on the device
  circuit  a brickwork circuit from |0...0>, one update after another
  batch    an ensemble of circuits, one program for all of them
  mpo      an operator applied to a chain, which is then compressed
  split    contract_svd on host tensors
  chain    a network of neighbouring site tensors contracted to one tensor
  expect   expectation values along a chain
"""

import math
import os

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DTYPES = {"c64": np.complex64, "c128": np.complex128}


def listed():
    return [
        # the benchmark's bond: 1024 states, mixed precision, rank held by the cap
        {"name": "bond c64 1024", "kind": "bond", "op": "gate", "dtype": "c64", "chil": 1024, "chim": 1024,
         "chir": 1024, "chi_max": 1024, "decay": 0.97},
        # the middle of the single-bond sweep
        {"name": "bond c64 256", "kind": "bond", "op": "gate", "dtype": "c64", "chil": 256, "chim": 256,
         "chir": 256, "chi_max": 256, "decay": 0.9},
        # the smallest call: an odd bond near a chain's end, where launches count
        {"name": "bond c64 37x45x51", "kind": "bond", "op": "gate", "dtype": "c64", "chil": 37, "chim": 45,
         "chir": 51, "chi_max": 40, "decay": 0.85},
        # the plain FP64 update of the single-bond sweep's smallest bond
        {"name": "bond c128 64", "kind": "bond", "op": "gate", "dtype": "c128", "chil": 64, "chim": 64,
         "chir": 64, "chi_max": 64, "decay": 0.97},
        # the 12-qubit circuit of the parity workload
        {"name": "circuit c128 12", "kind": "circuit", "dtype": "c128", "n": 12, "depth": 8, "chi_max": 32,
         "cutoff": 1e-10},
        # the same kind of circuit in mixed precision, at its full rank
        {"name": "circuit c64 14", "kind": "circuit", "dtype": "c64", "n": 14, "depth": 10, "chi_max": 128,
         "cutoff": 1e-8},
        # many small circuits of Haar gates, a new program on each call
        {"name": "batch haar 200", "kind": "batch", "gates": "haar", "circuits": 200, "n_lo": 6, "n_hi": 11,
         "depth_lo": 4, "depth_hi": 12, "replay": False, "cutoff": 1e-8},
        # the serving-style ensemble: uneven qubits, depths and caps, the captured program replayed
        {"name": "batch ising 64", "kind": "batch", "gates": "ising", "circuits": 64, "n_lo": 8, "n_hi": 40,
         "depth_lo": 4, "depth_hi": 12, "replay": True, "cutoff": 1e-5},
        # a step of the operator workload: transverse-field Ising MPO, compression, energy
        {"name": "mpo c64 18x80", "kind": "mpo", "dtype": "c64", "n": 18, "chi": 80, "decay": 0.93},
        # the reference's contract_svd on two site tensors
        {"name": "split c128 200x120x210", "kind": "split", "dtype": "c128", "d1": 200, "dm": 120, "d2": 210,
         "er": 1e-9},
        # four neighbouring sites contracted to one tensor, the network path on the tensor cores
        {"name": "chain c64 4x300", "kind": "chain", "dtype": "c64", "sites": 4, "chil": 300, "chim": 288,
         "chir": 310},
        # <ZZ> on every bond of a chain
        {"name": "expect c64 16x128", "kind": "expect", "dtype": "c64", "n": 16, "chi": 128, "decay": 0.95},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _near(rng, v):
    return max(2, int(v * rng.uniform(0.75, 1.0)))


def draw(rng):
    kind = rng.choice(["bond", "bond", "bond", "circuit", "batch", "mpo", "split", "chain", "expect"])
    dtype = rng.choice(["c64", "c128"])
    if kind == "bond":
        op = rng.choice(["gate", "gate", "switch"])
        # the FP64 split serves complex128 bonds and every switch
        chim = _log(rng, 16, 1000) if dtype == "c64" and op == "gate" else _log(rng, 8, 160 if op == "gate" else 90)
        return {"kind": kind, "op": op, "dtype": dtype, "chil": _near(rng, chim), "chim": chim,
                "chir": _near(rng, chim), "chi_max": max(2, int(chim * rng.uniform(0.6, 1.0))) if op == "gate" else 0,
                "decay": math.exp(-rng.uniform(24, 32) / max(chim, 32))}
    if kind == "circuit":
        n = rng.randint(6, 12)
        return {"kind": kind, "dtype": dtype, "n": n, "depth": rng.randint(4, 10),
                "chi_max": 32 if dtype == "c128" else 1 << ((n + 1) // 2), "cutoff": rng.choice([1e-8, 1e-10])}
    if kind == "batch":
        gates = rng.choice(["haar", "ising"])
        n_lo = rng.randint(4, 8)
        return {"kind": kind, "gates": gates, "circuits": _log(rng, 16, 200 if gates == "haar" else 60),
                "n_lo": n_lo, "n_hi": rng.randint(n_lo, 11 if gates == "haar" else 40), "depth_lo": 4,
                "depth_hi": rng.randint(4, 11), "replay": rng.random() < 0.5,
                "cutoff": 1e-8 if gates == "haar" else 1e-5}
    if kind == "mpo":
        return {"kind": kind, "dtype": "c64", "n": rng.randint(8, 17), "chi": _log(rng, 12, 76),
                "decay": rng.uniform(0.88, 0.93)}
    if kind == "split":
        dm = _log(rng, 8, 110)
        return {"kind": kind, "dtype": dtype, "d1": _near(rng, 2 * dm), "dm": dm, "d2": _near(rng, 2 * dm),
                "er": 1e-9}
    if kind == "chain":
        chi = _log(rng, 12, 384 if dtype == "c64" else 192)
        return {"kind": kind, "dtype": dtype, "sites": rng.randint(2, 4), "chil": _near(rng, chi), "chim": chi,
                "chir": _near(rng, chi)}
    return {"kind": kind, "dtype": dtype, "n": rng.randint(6, 16), "chi": _log(rng, 8, 120),
            "decay": rng.uniform(0.8, 0.95)}


# ---------------------------------------------------------------------------
# inputs, on the host, from the seed alone
# ---------------------------------------------------------------------------

def _gauss(rng, shape, dtype):
    real = np.float32 if dtype == np.complex64 else np.float64
    return rng.standard_normal(shape, real) + 1j * rng.standard_normal(shape, real)


def _isometry(rng, rows, cols, dtype):
    return np.linalg.qr(_gauss(rng, (rows, cols), dtype))[0]


def _haar(rng, count):
    q, r = np.linalg.qr(_gauss(rng, (count, 4, 4), np.complex128))
    d = np.einsum("tii->ti", r)
    return q * (d / np.abs(d))[:, None, :]


_PAULI = {"I": np.eye(2), "X": np.array([[0.0, 1.0], [1.0, 0.0]]), "Z": np.diag([1.0, -1.0])}


def _ising(rng, count):
    """exp(-i dt (J ZZ + hx X + hz Z)) gates of a disordered Ising chain."""
    k = np.kron
    zz, x = k(_PAULI["Z"], _PAULI["Z"]), k(_PAULI["X"], _PAULI["I"]) + k(_PAULI["I"], _PAULI["X"])
    z = k(_PAULI["Z"], _PAULI["I"]) + k(_PAULI["I"], _PAULI["Z"])
    j, hx, hz = rng.uniform(0.5, 1.5, (3, count, 1, 1))
    w, v = np.linalg.eigh(j * zz + 0.5 * hx * x + 0.25 * hz * z)
    return (v * np.exp(-0.3j * w)[:, None, :]) @ v.transpose(0, 2, 1)


def _brickwork(n, depth):
    """(layer, wire) pairs, wires from 1."""
    return [(layer, w) for layer in range(depth) for w in range(1 + layer % 2, n, 2)]


def _decaying(rng, n, chi, decay, dtype):
    """A chain of n sites whose bond spectra fall as decay^k."""
    dims = [min(2 ** i, 2 ** (n - i), chi) for i in range(n + 1)]
    sites = []
    for i in range(n):
        q = _isometry(rng, 2 * dims[i], dims[i + 1], dtype)
        s = decay ** np.arange(dims[i + 1])
        sites.append((q * (s / np.linalg.norm(s))).astype(dtype).reshape((dims[i], 2, dims[i + 1]), order="F"))
    return sites


def _ising_mpo(rng, n):
    """Sites (b, out, in, b') of sum Z Z + h_i X."""
    h = rng.uniform(0.5, 1.5, n)
    mpo = []
    for i in range(n):
        w = np.zeros((3, 2, 2, 3), np.complex128)
        w[0, :, :, 0] = w[2, :, :, 2] = _PAULI["I"]
        w[1, :, :, 0] = w[2, :, :, 1] = _PAULI["Z"]
        w[2, :, :, 0] = h[i] * _PAULI["X"]
        w = w[2:] if i == 0 else w
        mpo.append(np.asfortranarray(w[..., :1] if i == n - 1 else w))
    return mpo


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    dtype = DTYPES[case.get("dtype", "c64")]
    if kind == "bond":
        cl, cm, cr = case["chil"], case["chim"], case["chir"]
        s = case["decay"] ** np.arange(cm)
        s /= np.linalg.norm(s)
        a = (_isometry(rng, max(2 * cl, cm), cm, dtype)[:2 * cl] * s).astype(dtype)
        b = _isometry(rng, max(2 * cr, cm), cm, dtype)[:2 * cr].conj().T.astype(dtype)
        gate = _haar(rng, 1)[0] if case["op"] == "gate" else np.eye(4)[[0, 2, 1, 3]]
        return {"a": a.reshape((cl, 2, cm), order="F"), "b": b.reshape((cm, 2, cr), order="F"), "s": s, "gate": gate}
    if kind == "circuit":
        where = _brickwork(case["n"], case["depth"])
        return {"gates": list(zip((w for _, w in where), _haar(rng, len(where))))}
    if kind == "batch":
        lo, hi = case["n_lo"], case["n_hi"]
        n = rng.integers(lo, hi + 1, case["circuits"])
        depth = rng.integers(case["depth_lo"], case["depth_hi"] + 1, case["circuits"])
        if case["gates"] == "haar":  # caps at the circuits' full rank: 16 to 64
            cap = np.maximum(16, 2 ** ((n + 1) // 2))
        else:
            cap = rng.choice([16, 32, 64, 128], case["circuits"])
        layers = [[] for _ in range(int(depth.max()))]
        for c in range(case["circuits"]):
            where = _brickwork(int(n[c]), int(depth[c]))
            for (layer, w), g in zip(where, (_haar if case["gates"] == "haar" else _ising)(rng, len(where))):
                layers[layer].append((c, w, g))
        return {"n": n, "cap": cap, "layers": layers}
    if kind == "mpo":
        return {"sites": _decaying(rng, case["n"], case["chi"], case["decay"], dtype), "mpo": _ising_mpo(rng, case["n"])}
    if kind == "expect":
        return {"sites": _decaying(rng, case["n"], case["chi"], case["decay"], dtype)}
    if kind == "split":
        return {"t1": np.asfortranarray(_gauss(rng, (case["d1"], 2, case["dm"]), dtype)),
                "t2": np.asfortranarray(_gauss(rng, (case["dm"], 2, case["d2"]), dtype))}
    dims = [case["chil"]] + [case["chim"]] * (case["sites"] - 1) + [case["chir"]]
    return {"sites": [np.asfortranarray(_gauss(rng, (dims[i], 2, dims[i + 1]), dtype)) for i in range(case["sites"])]}


# ---------------------------------------------------------------------------
# through the framework
# ---------------------------------------------------------------------------

_engines = {}


def _framework():
    from __graft_entry__ import load_package
    return load_package()


def _engine(mode):
    """The engine of a program: one for each mode, kept for its calls."""
    if mode not in _engines:
        qt = _framework()
        eng = qt.Engine(mode=mode, tc_gemm=1) if mode == "chosen" else qt.Engine(mode=mode)
        if mode == "chosen":
            eng.set_rank_params(np.load(os.path.join(ROOT, "qaintensor.jl_gb300", "rank_model_params.npy")))
        _engines[mode] = eng
    return _engines[mode]


def prepare(case, seed):
    dtype = DTYPES[case.get("dtype", "c64")]
    eng = _engine("chosen" if dtype == np.complex64 else "plain")
    state = dict(case, eng=eng, **_inputs(case, seed))
    if case["kind"] == "bond":
        state["mps"] = eng.mps([state["a"], state["b"]], dtype=dtype)
        state["mps"].set_bond_spectrum(1, state["s"])
    elif case["kind"] in ("mpo", "expect"):
        state["mps"] = eng.mps(state["sites"], dtype=dtype)
    elif case["kind"] == "batch":
        state["batch"] = _framework().Batch(eng, state["n"], state["cap"])
        if case["replay"]:
            state["batch"].run(state["layers"], case["cutoff"])
    return state


def _amplitudes(eng, sites):
    """A chain's tensors contracted to one tensor with every open leg."""
    n = len(sites)
    bonds = [[(i, 3), (i + 1, 1)] for i in range(1, n)]
    legs = [(1, 1)] + [(i, 2) for i in range(1, n + 1)] + [(n, 3)]
    return _framework().contract(eng, sites, bonds, legs)


def run(state):
    eng, kind = state["eng"], state["kind"]
    if kind == "bond":
        mps = state["mps"].clone()
        if state["op"] == "gate":
            mps.apply_2q(state["gate"], 1, 1e-6, state["chi_max"])
        else:
            mps.switch(1)
        a, b = mps.site(1), mps.site(2)
        mps.free()
        return {"pair": eng.contract_pair(a, b, [2], [0]), "rank": a.shape[2]}
    if kind == "circuit":
        mps = eng.product_state(state["n"], dtype=DTYPES[state["dtype"]])
        ranks = [mps.apply_2q(g, w, state["cutoff"], state["chi_max"])["rank"] for w, g in state["gates"]]
        psi = _amplitudes(eng, mps.sites())
        mps.free()
        return {"amplitudes": psi, "ranks": np.array(ranks)}
    if kind == "batch":
        batch = state["batch"]
        batch.reset()
        if state["replay"]:
            batch.replay()
        else:
            batch.run(state["layers"], state["cutoff"])
        # complex64 states: their expectation values are kept as 32-bit numbers
        z = [batch.expect_z(i).astype(np.float32) for i in range(1, int(state["n"].min()) + 1)]
        # ranks that the cutoff decides within 32-bit rounding are not results to rely on
        full = state["gates"] == "haar"
        return {"z": z, "bonds": np.concatenate([batch.bond_dims(c) for c in range(len(state["n"]))]) if full else None}
    if kind == "mpo":
        mps = state["mps"].clone()
        mps.apply_mpo(state["mpo"])
        ranks, _ = mps.compress(1e-9, state["chi"], mode="chosen")
        energy = mps.expect_mpo(state["mpo"])
        psi = _amplitudes(eng, mps.sites())
        mps.free()
        return {"amplitudes": psi, "energy": np.float32(energy), "ranks": ranks}
    if kind == "split":
        return eng.contract_svd(state["t1"], state["t2"], (3, 1), state["er"])
    if kind == "chain":
        return _amplitudes(eng, state["sites"])
    zz = np.array([state["mps"].expect_zz(i) for i in range(1, state["n"])])
    return {"zz": zz, "norm2": np.float64(state["mps"].norm2())}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _split_flops(m, n, k):
    """A rank-k split of an m x n matrix: its products with a basis of k vectors, twice."""
    return 16.0 * m * n * k


def work(case):
    kind = case["kind"]
    size = 16 if case.get("dtype") == "c128" else 8
    if kind == "bond":
        cl, cm, cr = case["chil"], case["chim"], case["chir"]
        k = case["chi_max"] or min(2 * cl, 2 * cr)
        return {"bytes": size * (2.0 * cl * cm + 2.0 * cm * cr + 4.0 * cl * cr),
                "flops": 32.0 * cl * cm * cr + 128.0 * cl * cr + _split_flops(2 * cl, 2 * cr, k)}
    if kind == "circuit":
        flops = 0.0
        for _, w in _brickwork(case["n"], case["depth"]):
            d = [min(2 ** i, 2 ** (case["n"] - i), case["chi_max"]) for i in (w - 1, w, w + 1)]
            flops += 32.0 * d[0] * d[1] * d[2] + _split_flops(2 * d[0], 2 * d[2], d[1])
        return {"bytes": size * 2.0 ** case["n"], "flops": flops}
    if kind == "batch":
        n, depth = (case["n_lo"] + case["n_hi"]) / 2, (case["depth_lo"] + case["depth_hi"]) / 2
        d = 2.0 ** (n / 2 - 1) if case["gates"] == "haar" else 16.0
        return {"bytes": case["circuits"] * n * 16 * d * d,
                "flops": case["circuits"] * n / 2 * depth * (32.0 * d ** 3 + _split_flops(2 * d, 2 * d, d))}
    if kind == "mpo":
        n, chi = case["n"], float(case["chi"])
        return {"bytes": size * (n * 4 * chi ** 2 + 2.0 ** n),
                "flops": n * (16 * 9 * 4 * chi ** 3 + _split_flops(2 * chi, 3 * chi, chi))}
    if kind == "split":
        d1, dm, d2 = 2.0 * case["d1"], case["dm"], 2.0 * case["d2"]
        return {"bytes": size * (d1 * dm + dm * d2 + d1 * d2),
                "flops": _split_flops(d1, dm, dm) + _split_flops(dm, d2, dm) + 8 * d1 * dm * d2}
    if kind == "chain":
        flops, left, read = 0.0, 2.0 * case["chil"], 2.0 * case["chil"] * case["chim"]
        for i in range(1, case["sites"]):
            right = case["chir"] if i == case["sites"] - 1 else case["chim"]
            flops += 8 * left * case["chim"] * 2 * right
            read += 2.0 * case["chim"] * right
            left *= 2
        return {"bytes": size * (read + left * case["chir"]), "flops": flops}
    n, chi = case["n"], float(case["chi"])
    return {"bytes": size * n * 2 * chi ** 2, "flops": (n - 1) * n * 32 * chi ** 3}


# ---------------------------------------------------------------------------
# in 64 bits
# ---------------------------------------------------------------------------

def _split64(m, cutoff, chi_max):
    """Truncated split: the smallest values whose norm stays within the cutoff are dropped."""
    u, s, vh = np.linalg.svd(m, full_matrices=False)
    above = np.nonzero(np.sqrt(np.cumsum(s[::-1] ** 2)) > cutoff)[0]
    k = max(1, len(s) - int(above[0])) if len(above) else 1
    k = min(k, chi_max) if chi_max > 0 else k
    return u[:, :k], s[:k, None] * vh[:k]


def _update64(a, b, gate, cutoff, chi_max):
    cl, cm, cr = a.shape[0], a.shape[2], b.shape[2]
    pair = (a.reshape((2 * cl, cm), order="F") @ b.reshape((cm, 2 * cr), order="F")).reshape((cl, 2, 2, cr), order="F")
    pair = np.einsum("pqrs,arsb->apqb", gate.reshape((2, 2, 2, 2), order="F"), pair)
    if cutoff is None:
        return pair, None
    u, v = _split64(pair.reshape((2 * cl, 2 * cr), order="F"), cutoff, chi_max)
    return u.reshape((cl, 2, -1), order="F"), v.reshape((-1, 2, cr), order="F")


def _amplitudes64(sites):
    t = sites[0]
    for s in sites[1:]:
        t = np.tensordot(t, s, 1)
    return t


def _expect64(sites, ops):
    """<psi| prod of one-site diagonals |psi>, {site: diagonal} in ops."""
    env = np.eye(sites[0].shape[0], dtype=np.complex128)
    for i, a in enumerate(sites):
        b = a * ops[i][None, :, None] if i in ops else a
        env = np.tensordot(a.conj(), np.tensordot(env, b, 1), ([0, 1], [0, 1]))
    return float(np.trace(env).real)


def _energy64(sites, mpo):
    env = np.eye(sites[0].shape[0], dtype=np.complex128)[:, None, :]
    for a, w in zip(sites, mpo):
        env = np.tensordot(a.conj(), np.einsum("bsuc,xbud->xscd", w, np.tensordot(env, a, 1)), ([0, 1], [0, 1]))
    return float(np.trace(env[:, 0, :]).real)


def _applied64(sites, mpo):
    return [np.einsum("bsuc,aud->basdc", w, a).transpose(0, 1, 2, 4, 3).reshape(
        (w.shape[0] * a.shape[0], 2, -1)) for a, w in zip(sites, mpo)]


def _compressed64(sites, cutoff, chi_max):
    sites = list(sites)
    n = len(sites)
    for i in range(n - 1):
        q, r = np.linalg.qr(sites[i].reshape(-1, sites[i].shape[2]))
        sites[i] = q.reshape(sites[i].shape[0], 2, -1)
        sites[i + 1] = np.tensordot(r, sites[i + 1], 1)
    sites[-1] = sites[-1] / np.linalg.norm(sites[-1])
    ranks = np.zeros(n - 1, np.int32)
    for i in range(n - 1, 0, -1):
        u, v = _split64(sites[i].reshape(sites[i].shape[0], -1).conj().T, cutoff, chi_max)
        ranks[i - 1] = u.shape[1]
        sites[i - 1] = np.tensordot(sites[i - 1], v.conj().T, 1)
        sites[i] = u.conj().T.reshape(-1, 2, sites[i].shape[2])
    return sites, ranks


def exact(case, seed):
    kind = case["kind"]
    x = _inputs(case, seed)
    wide = lambda ts: [np.asarray(t, np.complex128) for t in ts]  # noqa: E731
    if kind == "bond":
        a, b = wide([x["a"], x["b"]])
        if case["op"] == "switch":
            return {"pair": _update64(a, b, x["gate"], None, 0)[0], "rank": None}
        a, b = _update64(a, b, x["gate"], 1e-6, case["chi_max"])
        return {"pair": np.tensordot(a, b, 1), "rank": a.shape[2]}
    if kind == "circuit":
        sites = [np.array([1.0, 0.0], np.complex128).reshape(1, 2, 1) for _ in range(case["n"])]
        ranks = []
        for w, g in x["gates"]:
            sites[w - 1], sites[w] = _update64(sites[w - 1], sites[w], g, case["cutoff"], case["chi_max"])
            ranks.append(sites[w].shape[0])
        return {"amplitudes": _amplitudes64(sites), "ranks": np.array(ranks)}
    if kind == "batch":
        if case["gates"] != "haar":
            return None  # hundreds of truncated splits of up to 256 x 256 a circuit
        psi = [np.zeros((2,) * int(n), np.complex128) for n in x["n"]]
        for p in psi:
            p[(0,) * p.ndim] = 1.0
        for layer in x["layers"]:
            for c, w, g in layer:
                t = np.tensordot(g.reshape((2, 2, 2, 2), order="F"), psi[c], ([2, 3], [w - 1, w]))
                psi[c] = np.moveaxis(t, (0, 1), (w - 1, w))
        out = []
        for i in range(int(x["n"].min())):
            p = [np.sum(np.abs(np.moveaxis(t, i, 0).reshape(2, -1)) ** 2, axis=1) for t in psi]
            out.append(np.array([(q[0] - q[1]) / (q[0] + q[1]) for q in p]))
        return {"z": out, "bonds": None}
    if kind == "mpo":
        sites, ranks = _compressed64(_applied64(wide(x["sites"]), x["mpo"]), 1e-9, case["chi"])
        return {"amplitudes": _amplitudes64(sites), "energy": _energy64(sites, x["mpo"]) / _expect64(sites, {}),
                "ranks": ranks}
    if kind == "split":
        t1, t2 = wide([x["t1"], x["t2"]])
        u1, v1 = _split64(t1.reshape((-1, case["dm"]), order="F"), case["er"], 0)
        u2, v2 = _split64(t2.reshape((case["dm"], -1), order="F"), case["er"], 0)
        return (u1 @ v1 @ u2 @ v2).reshape((case["d1"], 2, 2, case["d2"]), order="F")
    if kind == "chain":
        return _amplitudes64(wide(x["sites"]))
    sites, z = wide(x["sites"]), np.array([1.0, -1.0])
    norm2 = np.float64(_expect64(sites, {}))
    return {"zz": np.array([_expect64(sites, {i: z, i + 1: z}) for i in range(case["n"] - 1)]) / norm2, "norm2": norm2}
