"""The FP64 form on the tensor cores (U columns in 7 limbs, y' in 8) against the
long-double oracle and the CUDA-core kernel: limb widths from the narrowest to
the widest, short and long rows, heavy-tailed phenotypes, missing samples.

Bounds.  A column's limbs hold it to half a unit of 2^-54 (U) or 2^-62 (y') of
its largest value, the sums are exact and rounded once, and the operands are
doubles themselves; so U'x and x.y' are good to a few roundings of their terms:
|xxM - exact| <= (k + 8) 2^-52 c and |xyM - exact| <= 2^-50 ||y - mean|| sqrt(c)
with c = popcount(x)."""
import numpy as np
import pytest

from oracle import oracle as O
from supergwas_b200 import api, synth
from test_gpu_ts_shapes import awkward_rows

pytestmark = pytest.mark.gpu

SHAPES = [(1, 0, 40), (64, 2, 129), (200, 6, 20_001), (640, 18, 3000), (1000, 11, 40_000), (1000, 19, 2000),
          (1500, 28, 1500), (2000, 33, 19_001), (2600, 36, 700), (5000, 20, 1200), (900, 40, 500)]


@pytest.mark.parametrize("n,k,m", SHAPES, ids=lambda v: str(v))
@pytest.mark.parametrize("tail", [False, True])
def test_limbs_match_long_double_oracle(built, n, k, m, tail, monkeypatch):
    rng = np.random.default_rng(n + k)
    pop = np.arange(n) * 4 // n
    Z = rng.standard_normal((n, k))
    if k:
        Z[:, 0] = 1.0
    for s in range(1, min(4, k)):
        Z[:, s] = pop == s
    U = np.linalg.qr(Z)[0] if k else np.zeros((n, 0))
    y = rng.standard_cauchy(n) * 1e3 if tail else rng.standard_normal(n) + 0.5 * pop + 3.0
    x = awkward_rows(n, m, pop, y, rng)
    X = synth.pack_rows(x)
    o = O.cols_stats(X, n, U, y, 0.0)
    with api.Kgwas(precision="fp64", corr_threshold=0.0, log10_thresh=2.0) as g:
        g.set_structure(U, y)
        res, hits = g.run_host(X, stats=True), g.run_host(X).hits
        assert g.last_kernel() == "fp64"
        monkeypatch.setenv("KG_KERNEL", "fp64cores")
        cores = g.run_host(X, stats=True)
    st = res.stats
    assert np.array_equal(st["tested"], o["tested"]) and res.n_tested == o["n_tested"]
    assert np.array_equal(hits, res.hits)
    assert np.array_equal(hits["kmer"], cores.hits["kmer"])
    t = o["tested"]
    c = x.sum(axis=1, dtype=np.int64)[t].astype(float)
    assert np.all(np.abs(st["xxM"][t] - o["xxM"][t]) <= (k + 8) * 2.0**-52 * c)
    assert np.all(np.abs(st["xyM"][t] - o["xyM"][t]) <= 2.0**-50 * np.linalg.norm(y - y.mean()) * np.sqrt(c))


@pytest.mark.parametrize("thr,lt", [(0.0, 6.0), (0.2, 1.0), (0.2, 4.0)])
@pytest.mark.parametrize("n,k", [(700, 9), (1000, 25)])
def test_screen_keeps_counts_and_rows(built, n, k, thr, lt):
    """Without per-k-mer outputs the screen decides most k-mers; rows hold
    samples without a phenotype."""
    rng = np.random.default_rng(n * k)
    pop = np.arange(n) * 5 // n
    keep = np.sort(rng.choice(n, n - n // 9, replace=False))
    Z = rng.standard_normal((n, k))
    Z[:, 0] = 1.0
    for s in range(1, 5):
        Z[:, s] = pop == s
    U = np.linalg.qr(Z[keep])[0]
    y = rng.standard_normal(n) + 0.5 * pop
    X = synth.pack_rows(awkward_rows(n, 30_000, pop, y, rng))
    with api.Kgwas(precision="fp64", corr_threshold=thr, log10_thresh=lt) as g:
        g.set_structure(U, y[keep], keep, n)
        a, b = g.run_host(X, stats=True), g.run_host(X)
    assert a.hits.shape[0] > 0
    assert a.n_tested == b.n_tested
    assert np.array_equal(a.hits, b.hits)
