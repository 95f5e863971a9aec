"""Pair test of a phenotype whose yyM is rounding noise (src/kgwas_2d.cpp:292-318
asks for yyM > 1e-12): no pair counts as evaluated, on either kernel."""
import numpy as np
import pytest

from supergwas_b200 import api, synth
from test_gpu_screen4 import structure
from test_gpu_ts_shapes import awkward_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,evaluated", [(1e-9, False), (1e-6, True)])
def test_small_phenotypes(built, scale, evaluated, monkeypatch):
    n, k, m = 1000, 17, 300
    rng = np.random.default_rng(5)
    pop, Z = structure(n, k, rng)
    U, y = np.linalg.qr(Z)[0], scale * (rng.standard_normal(n) + 0.5 * pop)
    assert (np.sum(y * y) - np.sum((U.T @ y) ** 2) > 1e-12) == evaluated
    X = synth.pack_rows(awkward_rows(n, m, pop, y, rng))
    with api.Kgwas(corr_threshold=0.0, log10_thresh=6.0) as g:
        g.set_structure(U, y)
        out = []
        for kern in (None, "full"):
            monkeypatch.setenv("KG_KERNEL", kern) if kern else monkeypatch.delenv("KG_KERNEL", raising=False)
            out.append(g.run_pairs_host(X))
    assert out[0][1] == out[1][1]
    assert np.array_equal(out[0][0], out[1][0])
    assert (out[0][1] > 0) == evaluated
    if not evaluated:
        assert out[0][0].shape[0] == 0
