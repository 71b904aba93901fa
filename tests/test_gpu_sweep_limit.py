"""The sweep limit of FP32 splits whose sweeps run in one launch: the rule that
accepts a split out of sweeps looks at its last sweep alone, as it does with
one launch per sweep (which the trace asks for).  Spectra with a well separated
upper part and a plateau near the rounding level, whose columns still rotate
when the upper ones have converged: small limits that end in an error, in an
accepted split and in a converged one, with the same bits either way."""
import hashlib
import json
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHAPES = [(96, 80, 20, 3e-6), (160, 128, 30, 2e-6), (64, 100, 20, 2e-6)]
LIMITS = [6, 8, 10, 12, 80]


def outcomes(engine):
    out = []
    for (m, n, big, low) in SHAPES:
        rng = np.random.default_rng(m)
        k = min(m, n)
        q1 = np.linalg.qr(rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k)))[0]
        q2 = np.linalg.qr(rng.standard_normal((n, k)) + 1j * rng.standard_normal((n, k)))[0]
        s = np.concatenate([np.linspace(1, 0.3, big), np.full(k - big, low)])
        M = ((q1 * s) @ q2.conj().T).astype(np.complex64)
        # just above the FP32 resolution, too low for the fast freeze
        cut = 1.05 * 4 * np.sqrt(max(m, n)) * 5.96e-8 * np.linalg.norm(s)
        for limit in LIMITS:
            eng = engine.Engine(mode="chosen", max_sweeps=limit)
            try:
                U, S, Vh, rank, _ = eng.truncated_svd(M, cut, mode="chosen")
                left = eng.cert_counters()["fallback"]
                # (the FP64 split's orthonormalisation adds with atomics: its last bits vary)
                bits = "" if left else hashlib.sha256(U.tobytes() + S.tobytes() + Vh.tobytes()).hexdigest()
                out.append([m, limit, "ok", int(rank), left, bits])
            except engine.EngineError as e:
                out.append([m, limit, "error", int(e.code)])
            eng.close()
    return out


@pytest.mark.gpu
def test_sweep_limit_with_all_sweeps_in_one_launch(engine):
    env = dict(os.environ, QT_JACOBI_TRACE="1", PYTHONPATH=os.pathsep.join([ROOT, os.path.join(ROOT, "tests")]))
    r = subprocess.run([sys.executable, "-c", "import json, conftest, test_gpu_sweep_limit as t\n"
                        "print(json.dumps(t.outcomes(conftest.load_engine())))"],
                       env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    per_sweep = json.loads(r.stdout.strip().splitlines()[-1])
    assert outcomes(engine) == per_sweep
    # limits reached with only the plateau's columns still rotating, and accepted without the FP64 split
    assert [96, 10] in [o[:2] for o in per_sweep if o[2] == "ok" and o[4] == 0]
    assert [160, 12] in [o[:2] for o in per_sweep if o[2] == "ok" and o[4] == 0]
