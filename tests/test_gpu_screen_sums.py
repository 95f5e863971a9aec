"""The 4-bit screen's sums.  A phenotype that its limbs hold exactly (values 1 and
6 of both signs, mean 0, no covariate but the intercept) leaves the screen a bound
of 1e-5 and the 1e-4 that its cut lies below the emit cut, so rows whose x.y' is a
few units from the cut, in sums of several thousand, are emitted only if the sums
are right to about 2e-4; and rows at the longest row that the screen takes."""
import numpy as np
import pytest

from oracle import oracle as O
from supergwas_b200 import api, synth
from test_gpu_screen4 import structure
from test_gpu_ts_shapes import awkward_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1024, 4096])
def test_rows_a_few_units_from_the_cut(built, n, monkeypatch):
    lt = 80.0 if n == 1024 else 300.0
    y = np.resize([1.0, -1.0, 6.0, -6.0], n)
    U = np.full((n, 1), n ** -0.5)  # a power of two
    c = n // 2
    cut = 10.0 ** -lt
    # x.y' at the cut for c = n / 2: xxM = n / 4, yyM = 18.5 n
    from scipy import optimize, special
    chi = optimize.brentq(lambda t: special.log_ndtr(-np.sqrt(t)) + np.log(2.0) + lt * np.log(10.0), 1.0, 1e4)
    at = np.sqrt(-np.expm1(-chi / n) * (n / 4) * 18.5 * n)
    rng = np.random.default_rng(n)
    rows, xy = [], []
    for off in range(-30, 31):
        want = int(at) + off
        for sign in (1, -1):
            # ones and sixes with a net of `want`: a sixes more of one sign, then single units
            x = np.zeros(n, np.uint8)
            six, one = want // 6, want % 6
            pos = {v: rng.permutation(np.nonzero(y == v * sign)[0]) for v in (1, -1, 6, -6)}
            base6, base1 = (c // 2 - six) // 2, (c // 2 - one) // 2
            for v, k in ((6, base6 + six), (-6, base6), (1, base1 + one), (-1, base1)):
                x[pos[v][:k]] = 1
            rows.append(x)
            xy.append(x @ y)
            rows.append(1 - x)
            xy.append((1 - x) @ y)
    x = np.array(rows)
    X = synth.pack_rows(x)
    o = O.cols_stats(X, n, U, y, 0.0)
    want = np.nonzero(o["pval"] <= cut)[0]
    assert 20 < want.size < x.shape[0] - 20
    monkeypatch.setenv("KG_DEDUP", "0")
    with api.Kgwas(corr_threshold=0.0, log10_thresh=lt) as g:
        g.set_structure(U, y)
        r = g.run_host(X)
        assert g.last_screen() == 1
        g.set_phenotypes([(U, y, np.arange(n))] * 3, n)
        tested, hits = g.run_multi_host(X)
        assert g.last_screen() == 1
    assert r.n_tested == x.shape[0] and np.all(tested == x.shape[0])
    assert np.array_equal(r.hits["kmer"].astype(np.int64), want)
    for p in range(3):
        assert np.array_equal(hits["kmer"][hits["pheno"] == p].astype(np.int64), want)


@pytest.mark.parametrize("n,screened", [(24_576, 1), (24_577, 0)])
def test_longest_rows(built, n, screened, monkeypatch):
    rng = np.random.default_rng(n)
    pop, Z = structure(n, 4, rng)
    U, y = np.linalg.qr(Z)[0], rng.standard_normal(n) + 0.5 * pop
    X = synth.pack_rows(awkward_rows(n, 1500, pop, y, rng))
    monkeypatch.setenv("KG_DEDUP", "0")
    with api.Kgwas(corr_threshold=0.0, log10_thresh=6.0) as g:
        g.set_structure(U, y)
        a = g.run_host(X)
        assert g.last_screen() == screened
        monkeypatch.setenv("KG_KERNEL", "full")
        b = g.run_host(X)
    assert b.hits.shape[0] > 0
    assert a.n_tested == b.n_tested and np.array_equal(a.hits, b.hits)
