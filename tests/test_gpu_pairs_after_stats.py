"""A call for every k-mer's statistics between two pair tests of one context."""
import numpy as np
import pytest

from supergwas_b200 import api
from test_gpu_screen_gives_up import batch

pytestmark = pytest.mark.gpu


def test_pairs_statistics_pairs(built):
    U, y, X = batch(1000, 17, 300, 0.1, np.random.default_rng(6))
    with api.Kgwas(corr_threshold=0.0, log10_thresh=6.0) as g:
        g.set_structure(U, y)
        a, ea = g.run_pairs_host(X)
        g.run_host(X, stats=True)
        b, eb = g.run_pairs_host(X)
    assert ea == eb > 0
    assert np.array_equal(a, b)
