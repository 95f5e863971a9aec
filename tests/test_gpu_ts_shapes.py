"""The tensor-memory kernel on rows shorter than one 128-byte TMA box row and on
limb images that nearly fill shared memory: bit for bit the smem-A kernel's
statistics (both sum the same integers and evaluate the same expressions)."""
import numpy as np
import pytest

from supergwas_b200 import api, synth

pytestmark = pytest.mark.gpu

# (samples, k-mers, principal components): row widths of 16, 32, ..., 112
# bytes, tiles of 1, 127, 128 and 129 k-mers and many tiles per SM, images of
# 128 KB and more
SHAPES = [(1, 50, 0), (64, 127, 3), (128, 128, 4), (129, 129, 5), (250, 60_001, 5), (300, 2049, 12), (500, 1, 6),
          (640, 20_000, 10), (700, 777, 32), (896, 3000, 16), (2000, 3001, 20), (1700, 40_000, 24)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "n%d_m%d_r%d" % s)
@pytest.mark.parametrize("thr", [0.0, 0.2])
def test_same_statistics_as_smem_kernel(built, shape, thr, monkeypatch):
    n, m, r = shape
    ds = synth.simulate(n=n, m=m, S=max(1, min(5, n // 2)), r=min(r, max(n - 1, 0)) if n > 1 else 0,
                        n_causal=min(3, m), missing=0.0, seed=500 + n)
    X = ds.packed_overlap()
    U = ds.U if r > 0 and n > 1 else np.zeros((ds.n, 0))
    out = {}
    for kern in ("ts", "ss"):
        monkeypatch.setenv("KG_KERNEL", kern)
        with api.Kgwas(corr_threshold=thr, log10_thresh=1.0) as g:
            g.set_structure(U, ds.y)
            out[kern] = g.run_host(X, stats=True), g.run_host(X)
            assert g.last_kernel() == kern
    for a, b in zip(out["ts"], out["ss"]):
        assert a.n_tested == b.n_tested
        assert np.array_equal(a.hits, b.hits)
    for f, v in out["ts"][0].stats.items():
        assert np.array_equal(v, out["ss"][0].stats[f]), f
