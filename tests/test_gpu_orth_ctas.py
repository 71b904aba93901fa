"""The one-launch FP32 orthonormalisation over its CTA counts (16 rows each):
one CTA, one and two partial sums per lane, four entries of the summed Gram
per warp at a time and one, through the compression of a chain whose norm
the orthonormal bases have to keep."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chi", [3, 33, 260, 530, 640])
def test_fp32_compression_keeps_the_norm(engine, chi):
    rng = np.random.default_rng(chi)
    n = 2 * int(np.ceil(np.log2(chi))) + 2
    dims = [min(2 ** i, 2 ** (n - i), chi) for i in range(n + 1)]
    sites = [((rng.standard_normal((dims[i], 2, dims[i + 1])) + 1j * rng.standard_normal((dims[i], 2, dims[i + 1])))
              / np.sqrt(4 * dims[i + 1])).astype(np.complex64) for i in range(n)]
    eng = engine.Engine(mode="chosen")
    mps = eng.mps(sites, dtype=np.complex64)
    before = mps.norm2()
    cutoff = 1e-4 * np.sqrt(before)  # above the FP32 resolution: no FP64 split
    mps.compress(cutoff, chi, mode="chosen", normalize=False)
    # each of 2 n steps leaves its basis orthonormal to FP32 rounding of sums of
    # 2 chi terms (a few u each), and drops at most cutoff^2
    bound = 2 * n * 4 * np.sqrt(2 * chi) * 5.96e-8 + n * 1e-8
    assert abs(mps.norm2() / before - 1) <= bound, (mps.norm2(), before, bound)
    mps.free()
    eng.close()
