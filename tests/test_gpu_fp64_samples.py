"""FP64 form at the largest cohorts: a phenotype whose low digits are all near
-128 (which enter as 128 x, every second sample) or 126 (as 64 x), so that the sum
of the four lowest limbs is as large as it gets.  Bound as in
test_gpu_fp64_limbs.py: |xyM - exact| <= 2^-50 ||y - mean|| sqrt(c)."""
import math

import numpy as np
import pytest

from oracle import oracle as O
from supergwas_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [10_880, 10_882, 12_288])
def test_largest_low_limb_sums(built, n):
    y = -np.where(np.arange(n) % 2 == 1, float(0x80808080), float(0x3F3F3F3F)) * 2.0 ** -61
    y[:2] = 1.0, -1.0
    y[-1] = -math.fsum(y[:-1])
    assert math.fsum(y) == 0.0
    rng = np.random.default_rng(n)
    x = (rng.random((130, n)) < np.linspace(0.5, 1.0, 130)[:, None]).astype(np.uint8)
    x[0] = 1
    x[:, [0, 1, n - 1]] = 0
    X = synth.pack_rows(x)
    o = O.cols_stats(X, n, np.zeros((n, 0)), y, 0.0)
    with api.Kgwas(precision="fp64", corr_threshold=0.0, log10_thresh=2.0) as g:
        g.set_structure(np.zeros((n, 0)), y)
        st = g.run_host(X, stats=True).stats
    c = x.sum(axis=1).astype(float)
    assert np.all(np.abs(st["xyM"] - o["xyM"]) <= 2.0 ** -50 * np.linalg.norm(y) * np.sqrt(c))
