"""FP64 form: an intercept column whose entries are off by a few units of their
last place, one sign per half of the samples.  The half's row meets the sum of
them: left out, it moves xxM by 2^-48 c.

Bound: a_0 and s_0 = a_0 c + e_0 are rounded once each, s_0^2 <= c and xxM once
more (6 x 2^-53 c together), and the limb that holds the entries leaves out at
most 1.6e-16 c."""
import numpy as np
import pytest

from oracle import oracle as O
from supergwas_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("units", [1, 16, 64])
def test_intercept_off_by_its_last_places(built, units):
    n = 1024
    half = np.arange(n) < n // 2
    rng = np.random.default_rng(units)
    U = (2.0 ** -5 * (1.0 + np.where(half, 1.0, -1.0) * units * 2.0 ** -52))[:, None]
    y = rng.standard_normal(n)
    x = (rng.random((200, n)) < 0.5).astype(np.uint8)
    x[0], x[1] = half, ~half
    x[2:100] &= half
    X = synth.pack_rows(x)
    o = O.cols_stats(X, n, U, y, 0.0)
    with api.Kgwas(precision="fp64", corr_threshold=0.0, log10_thresh=2.0) as g:
        g.set_structure(U, y)
        st = g.run_host(X, stats=True).stats
    c = x.sum(axis=1).astype(float)
    assert np.all(np.abs(st["xxM"] - o["xxM"]) <= 6 * 2.0 ** -53 * c + 1.6e-16 * c)
