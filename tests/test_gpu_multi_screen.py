"""The many-phenotype kernels with a resident image decide most (k-mer,
phenotype) tests in single precision; counts and rows must equal the streamed
kernel's, which evaluates the FP64 statistic for every one."""
import numpy as np
import pytest

from supergwas_b200 import api, synth
from test_gpu_ts_shapes import awkward_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("thr,lt", [(0.0, 6.0), (0.2, 1.0), (0.2, 6.0), (0.0, 3.0)])
@pytest.mark.parametrize("n,ks", [(300, (1, 3)), (300, (7, 2)), (900, (12, 15)), (1500, (22, 3)), (1200, (33, 41)),
                                  (700, (28, 30))], ids=lambda v: str(v))
def test_screened_tests_equal_streamed_kernel(built, n, ks, thr, lt, monkeypatch):
    rng = np.random.default_rng(n + ks[0])
    pop = np.arange(n) * 4 // n
    y0 = rng.standard_normal(n) + 0.5 * pop
    X = synth.pack_rows(awkward_rows(n, 9001, pop, y0, rng), max(16, synth.words_per_kmer(n)))
    phenos = []
    for p in range(5):
        keep = np.sort(rng.choice(n, n - p * n // 12, replace=False))
        Z = rng.standard_normal((n, ks[p % 2]))
        Z[:, 0] = 1.0
        for s in range(1, min(4, ks[p % 2])):
            Z[:, s] = pop == s
        U = np.linalg.qr(Z[keep])[0]
        phenos.append((U, ((y0 + 0.3 * rng.standard_normal(n)) * 10.0 ** (3 * p - 4))[keep], keep))
    shards = np.array([0, 100, 4000], dtype=np.uint64)
    out = {}
    for kern in ("mp", "mpb", "mpb2"):
        monkeypatch.setenv("KG_MP_KERNEL", kern)
        with api.Kgwas(corr_threshold=thr, log10_thresh=lt) as g:
            g.set_phenotypes(phenos, n)
            out[kern] = g.run_multi_host(X, shards)
    assert out["mp"][1].shape[0] > 0
    for kern in ("mpb", "mpb2"):
        assert np.array_equal(out[kern][0], out["mp"][0]), kern
        assert np.array_equal(out[kern][1], out["mp"][1]), kern
