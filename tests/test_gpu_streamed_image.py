"""The streamed-image kernel (limb images larger than shared memory) against
the smem-A kernel, bit for bit: one tile per item and two, odd tile counts,
rows that end inside a super-stage, an image chunk or a box, and the
single-precision screen against the FP64 statistic."""
import numpy as np
import pytest

from supergwas_b200 import api, synth
from test_gpu_ts_shapes import awkward_rows

pytestmark = pytest.mark.gpu

# (samples, U columns, k-mers)
SHAPES = [(2600, 41, 1), (2600, 41, 129), (2100, 35, 20_001), (2700, 30, 38_000), (4500, 17, 40_007), (5000, 33, 4000),
          (9000, 9, 2500), (3200, 41, 19_000)]


@pytest.mark.parametrize("n,k,m", SHAPES, ids=lambda v: str(v))
@pytest.mark.parametrize("thr,lt", [(0.0, 6.0), (0.2, 1.0)])
def test_streamed_image_equals_smem_kernel(built, n, k, m, thr, lt, monkeypatch):
    rng = np.random.default_rng(n + k + m)
    pop = np.arange(n) * 4 // n
    Z = rng.standard_normal((n, k))
    Z[:, 0] = 1.0
    for s in range(1, 4):
        Z[:, s] = pop == s
    U = np.linalg.qr(Z)[0]
    y = rng.standard_normal(n) + 0.5 * pop
    X = synth.pack_rows(awkward_rows(n, min(m, 4096), pop, y, rng))
    X = np.ascontiguousarray(X[np.arange(m) % X.shape[0]])
    monkeypatch.setenv("KG_DEDUP", "0")
    out = {}
    for kern in ("tb", "ss"):
        monkeypatch.setenv("KG_KERNEL", kern)
        with api.Kgwas(corr_threshold=thr, log10_thresh=lt) as g:
            g.set_structure(U, y)
            out[kern] = g.run_host(X, stats=m < 5000), g.run_host(X)
            assert g.last_kernel() == kern
    for a, b in zip(out["tb"], out["ss"]):
        assert a.n_tested == b.n_tested
        assert np.array_equal(a.hits, b.hits)
        for f in a.stats or {}:
            assert np.array_equal(a.stats[f], b.stats[f]), f
