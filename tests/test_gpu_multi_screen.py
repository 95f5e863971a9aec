"""The many-phenotype kernels decide most (k-mer, phenotype) tests in single
precision; counts and rows must equal those of the single-phenotype smem-A
kernel, which evaluates the FP64 statistic for every k-mer."""
import numpy as np
import pytest

from supergwas_b200 import api, synth
from test_gpu_ts_shapes import awkward_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("thr,lt", [(0.0, 6.0), (0.2, 1.0), (0.2, 6.0), (0.0, 3.0)])
@pytest.mark.parametrize("n,ks", [(300, (1, 3)), (300, (7, 2)), (900, (12, 15)), (1500, (22, 3)), (1200, (33, 41)),
                                  (700, (28, 30))], ids=lambda v: str(v))
def test_screened_tests_equal_smem_kernel(built, n, ks, thr, lt, monkeypatch):
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
    monkeypatch.setenv("KG_KERNEL", "ss")
    bounds = list(shards.astype(int)) + [X.shape[0]]
    total = 0
    for p, (U, y, keep) in enumerate(phenos):
        with api.Kgwas(corr_threshold=thr, log10_thresh=lt) as g:
            g.set_structure(U, y, keep, n)
            for s in range(3):
                ref = g.run_host(X[bounds[s]:bounds[s + 1]])
                total += ref.hits.shape[0]
                for kern, (tested, hits) in out.items():
                    assert tested[s, p] == ref.n_tested, (kern, p, s)
                    h = hits[(hits["pheno"] == p) & (hits["shard"] == s)]
                    assert np.array_equal(h["kmer"], ref.hits["kmer"] + np.uint64(bounds[s])), (kern, p, s)
                    for f in ("effect", "pval", "chisq"):
                        assert np.array_equal(h[f], ref.hits[f]), (kern, p, s, f)
            assert g.last_kernel() == "ss"
    assert total > 0
