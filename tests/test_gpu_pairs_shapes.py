"""The pair kernel where its schedule can go wrong -- several units and tiles
per CTA, super-stages that do not divide among the unpack groups, rows of one
to three boxes, images that leave no room for the rows i -- against the 1-D
test of the explicit product rows (the same exact sums and expressions)."""
import numpy as np
import pytest

from supergwas_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,m", [(1000, 17, 1500), (1300, 12, 900), (2000, 21, 700), (600, 30, 1100), (100, 3, 1501),
                                   (2500, 9, 600)], ids=lambda v: str(v))
@pytest.mark.parametrize("lt", [2.0, 6.0])
def test_pairs_equal_product_rows(built, n, k, m, lt):
    rng = np.random.default_rng(n + m)
    x = (rng.random((m, n)) < np.sin(0.5 * np.pi * rng.random((m, 1))) ** 2).astype(np.uint8)
    x[5], x[6], x[7] = 0, 1, x[8]
    Z = rng.standard_normal((n, k))
    Z[:, 0] = 1.0
    Z[:, 1] = np.arange(n) >= n // 3
    U = np.linalg.qr(Z)[0]
    y = rng.standard_normal(n) + 1.5 * (x[3] & x[9]) + 1.0 * (x[20] & x[m - 1]) + 3.0
    X = synth.pack_rows(x)
    ij = np.stack(np.triu_indices(m, 1), axis=1)
    with api.Kgwas(corr_threshold=0.0, log10_thresh=lt) as g:
        g.set_structure(U, y)
        for r0, r1 in ((0, m), (m // 3, m // 3 + 77)):
            pairs, evaluated = g.run_pairs_host(X, r0, r1)
            sel = ij[(ij[:, 0] >= r0) & (ij[:, 0] < r1)]
            res = g.run_host(np.ascontiguousarray(X[sel[:, 0]] & X[sel[:, 1]]))
            assert evaluated == res.n_tested
            hit = sel[res.hits["kmer"].astype(np.int64)]
            assert np.array_equal(pairs["a"], hit[:, 0].astype(np.uint64))
            assert np.array_equal(pairs["b"], hit[:, 1].astype(np.uint64))
            for f in ("effect", "pval", "chisq"):
                assert np.array_equal(pairs[f], res.hits[f]), f

