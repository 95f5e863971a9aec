"""KG_MP_STREAMED=1 takes the kernel with the streamed image also where the
4-bit screen would apply."""
import numpy as np
import pytest

from supergwas_b200 import api
from test_gpu_screen_gives_up import batch

pytestmark = pytest.mark.gpu


def test_streamed_image_is_taken(built, monkeypatch):
    n = 900
    rng = np.random.default_rng(4)
    U, y, X = batch(n, 12, 5000, 0.01, rng)
    phenos = [(U, y + 0.3 * rng.standard_normal(n), np.arange(n)) for _ in range(3)]
    out = []
    for streamed in (True, False):
        if streamed:
            monkeypatch.setenv("KG_MP_STREAMED", "1")
        else:
            monkeypatch.delenv("KG_MP_STREAMED")
        with api.Kgwas(corr_threshold=0.0, log10_thresh=6.0) as g:
            g.set_phenotypes(phenos, n)
            out.append(g.run_multi_host(X))
            assert g.multi_shape()["kernel"] == ("image streamed (mp)" if streamed else "4-bit screen (fs)")
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
