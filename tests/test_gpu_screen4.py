"""The 4-bit screen against the kernels that evaluate every k-mer: a row that
is emitted comes from the FP64 refinement on both sides, so counts and rows are
equal.  Row widths below and above one TMA box, rows that end inside a unit of
256 samples or a box, one and two limbs per U column, tiles of one row and many
per SM, and rows around every decision."""
import numpy as np
import pytest

from supergwas_b200 import api, synth
from test_gpu_ts_shapes import awkward_rows

pytestmark = pytest.mark.gpu

# (samples, U columns, k-mers)
SHAPES = [(64, 3, 129), (150, 2, 1), (200, 6, 60_001), (257, 5, 127), (640, 11, 20_000), (700, 9, 128),
          (1000, 17, 40_000), (1024, 30, 3000), (1025, 17, 3001), (2000, 21, 40_001), (2900, 33, 2500),
          (5000, 33, 20_000), (9000, 9, 2500)]


def structure(n, k, rng):
    pop = np.arange(n) * 4 // n
    Z = rng.standard_normal((n, k))
    Z[:, 0] = 1.0
    for s in range(1, min(4, k)):
        Z[:, s] = pop == s
    return pop, Z


def both(X, U, y, thr, lt, monkeypatch, kern, *where):
    monkeypatch.setenv("KG_DEDUP", "0")
    with api.Kgwas(corr_threshold=thr, log10_thresh=lt) as g:
        g.set_structure(U, y, *where)
        monkeypatch.delenv("KG_KERNEL", raising=False)
        a = g.run_host(X)
        monkeypatch.setenv("KG_KERNEL", kern)
        return a, g.run_host(X)


@pytest.mark.parametrize("n,k,m", SHAPES, ids=lambda v: str(v))
@pytest.mark.parametrize("thr,lt", [(0.0, 6.0), (0.2, 4.0), (1e-5, 9.0)])
def test_same_rows_as_full_kernel(built, n, k, m, thr, lt, monkeypatch):
    rng = np.random.default_rng(n + k + m)
    pop, Z = structure(n, k, rng)
    y = rng.standard_normal(n) + 0.5 * pop + 2.0
    X = synth.pack_rows(awkward_rows(n, min(m, 4096), pop, y, rng))
    X = np.ascontiguousarray(X[np.arange(m) % X.shape[0]])
    a, b = both(X, np.linalg.qr(Z)[0], y, thr, lt, monkeypatch, "full")
    assert a.n_tested == b.n_tested
    assert np.array_equal(a.hits, b.hits)
    if m > 2000:
        assert b.hits.shape[0] > 0


@pytest.mark.parametrize("tail", ["y", "U", "both", "scale"])
@pytest.mark.parametrize("thr", [0.0, 0.1])
def test_heavy_tails_and_missing_samples(built, tail, thr, monkeypatch):
    """Columns whose largest value is far above the rest leave the limbs less
    to hold the rest with; the bounds follow."""
    n, k, m = 1200, 12, 30_000
    rng = np.random.default_rng(len(tail))
    keep = np.sort(rng.choice(n, n - n // 7, replace=False))
    pop, Z = structure(n, k, rng)
    if tail in ("U", "both"):
        Z[:, 5:] = rng.standard_cauchy((n, k - 5))
    y = rng.standard_cauchy(n) if tail in ("y", "both") else rng.standard_normal(n) + 0.5 * pop
    U = np.linalg.qr(Z[keep])[0]
    if tail == "scale":
        U = U * 1.5  # not orthonormal: the general statistic
        y = y * 1e-9
    x = awkward_rows(n, m, pop, y, rng)
    a, b = both(synth.pack_rows(x), U, y[keep], thr, 4.0, monkeypatch, "full", keep, n)
    assert a.n_tested == b.n_tested
    assert np.array_equal(a.hits, b.hits)


@pytest.mark.parametrize("thr,lt", [(0.0, 6.0), (0.2, 4.0)])
@pytest.mark.parametrize("n,ks,np_", [(900, (12, 15), 5), (2000, (21, 3), 7), (1030, (5, 6), 17), (5000, (33, 30), 3),
                                      (300, (2, 3), 8)], ids=lambda v: str(v))
def test_many_phenotypes(built, n, ks, np_, thr, lt, monkeypatch):
    """Phenotypes of different widths and samples in one launch, several and
    single tiles per pass over the groups, shards that start inside a tile."""
    rng = np.random.default_rng(n + np_)
    pop, Z = structure(n, max(ks), rng)
    y0 = rng.standard_normal(n) + 0.5 * pop
    x = awkward_rows(n, 4096, pop, y0, rng)
    X = synth.pack_rows(np.concatenate([x] * 10)[:40_003], max(16, synth.words_per_kmer(n)))
    phenos = []
    for p in range(np_):
        keep = np.sort(rng.choice(n, n - p * n // 40, replace=False))
        U = np.linalg.qr(Z[keep][:, :ks[p % 2]])[0]
        phenos.append((U, (y0 + 0.3 * rng.standard_normal(n))[keep], keep))
    shards = np.array([0, 7, 100, 100, 20_000, 39_990], dtype=np.uint64)
    monkeypatch.setenv("KG_DEDUP", "0")
    out = []
    for kern, bt in (("mp", None), (None, None), (None, "1"), (None, "3")):
        for var, val in (("KG_MP_KERNEL", kern), ("KG_MP_BT", bt)):
            monkeypatch.setenv(var, val) if val else monkeypatch.delenv(var, raising=False)
        with api.Kgwas(corr_threshold=thr, log10_thresh=lt) as g:
            g.set_phenotypes(phenos, n)
            out.append(g.run_multi_host(X, shards))
            assert (g.multi_shape()["kernel"] == "4-bit screen (fs)") == (kern is None)
            if kern is None and bt is None:
                monkeypatch.setenv("KG_DEDUP", "1")
                out.append(g.run_multi_host(X, shards))
                monkeypatch.setenv("KG_DEDUP", "0")
    assert out[0][1].shape[0] > 0
    for tested, hits in out[1:]:
        assert np.array_equal(tested, out[0][0])
        assert np.array_equal(hits, out[0][1])


@pytest.mark.parametrize("n,k,m", [(1000, 17, 700), (300, 4, 1501), (2000, 21, 400), (1024, 9, 130)],
                         ids=lambda v: str(v))
@pytest.mark.parametrize("thr", [0.0, 0.2])
def test_pairs(built, n, k, m, thr, monkeypatch):
    rng = np.random.default_rng(n + m)
    pop, Z = structure(n, k, rng)
    y = rng.standard_normal(n) + 0.5 * pop
    x = awkward_rows(n, m, pop, y, rng)
    x[10:13] = 1  # products of all ones
    X = synth.pack_rows(x)
    with api.Kgwas(corr_threshold=thr, log10_thresh=4.0) as g:
        g.set_structure(np.linalg.qr(Z)[0], y)
        for r0, r1 in ((0, m), (m // 3, m // 3 + 33)):
            monkeypatch.delenv("KG_KERNEL", raising=False)
            a, ea = g.run_pairs_host(X, r0, r1)
            monkeypatch.setenv("KG_KERNEL", "full")
            b, eb = g.run_pairs_host(X, r0, r1)
            assert ea == eb
            assert np.array_equal(a, b)
        assert b.shape[0] > 0 or r1 < m


@pytest.mark.parametrize("n,k", [(200, 6), (1000, 33)])
def test_gate_decided_by_the_limb_sums(built, n, k, monkeypatch):
    """A correlation a few 1e-9 from the threshold, less than the roundings of
    the int8 limbs: the count of tested k-mers is that of the int8 kernels, for
    one phenotype and for many."""
    rng = np.random.default_rng(n)
    pop, Z = structure(n, k, rng)
    y = rng.standard_normal(n) + 1.5 * pop + 2.0
    U = np.linalg.qr(Z)[0]
    X = synth.pack_rows(awkward_rows(n, 2000, pop, y, rng), max(16, synth.words_per_kmer(n)))
    with api.Kgwas(corr_threshold=0.0, log10_thresh=6.0) as g:
        g.set_structure(U, y)
        st = g.run_host(X, stats=True).stats
    cor = np.abs(st["cor"])
    pick = rng.choice(np.nonzero((cor > 0.05) & (cor < 0.9))[0], 16, replace=False)
    for i, eps in zip(pick, [3e-9, -3e-9] * 8):
        with api.Kgwas(corr_threshold=float(cor[i] * (1 + eps)), log10_thresh=6.0) as g:
            g.set_structure(U, y)
            g.set_phenotypes([(U, y, np.arange(n))] * 2, n)
            monkeypatch.delenv("KG_KERNEL", raising=False)
            monkeypatch.delenv("KG_MP_KERNEL", raising=False)
            a, (ta, _) = g.run_host(X), g.run_multi_host(X)
            monkeypatch.setenv("KG_KERNEL", "full")
            monkeypatch.setenv("KG_MP_KERNEL", "mp")
            b, (tb, _) = g.run_host(X), g.run_multi_host(X)
        assert a.n_tested == b.n_tested
        assert np.array_equal(ta, tb) and ta[0, 0] == a.n_tested

@pytest.mark.parametrize("n,k,m,thr,lt", [(1000, 11, 420_001, 0.0, 6.0), (300, 12, 900_001, 0.2, 9.0),
                                          (2100, 21, 100_001, 0.2, 6.0), (1000, 11, 800_000, 0.0, 4.0)],
                         ids=lambda v: str(v))
def test_fp64_form(built, n, k, m, thr, lt, monkeypatch):
    """The FP64 form evaluates the rows that the screen leaves (gathered), or,
    where those are more than it has room for (the last case: every eighth row
    follows y), all rows."""
    rng = np.random.default_rng(n + m)
    pop, Z = structure(n, k, rng)
    y = rng.standard_normal(n) + 0.5 * pop
    x = awkward_rows(n, 4096, pop, y, rng)
    X = synth.pack_rows(x)
    X = np.ascontiguousarray(X[rng.integers(0, 4096, m)])
    if lt == 6.0:
        X[:, :] = X[np.where(np.arange(m) % 97 == 0, np.arange(m), np.arange(m) // 64 * 64 + 1)]
    monkeypatch.setenv("KG_DEDUP", "0")
    with api.Kgwas(precision="fp64", corr_threshold=thr, log10_thresh=lt) as g:
        g.set_structure(np.linalg.qr(Z)[0], y)
        monkeypatch.delenv("KG_KERNEL", raising=False)
        a, again = g.run_host(X), g.run_host(X)
        monkeypatch.setenv("KG_DEDUP", "1")
        runs = g.run_host(X)
        monkeypatch.setenv("KG_DEDUP", "0")
        monkeypatch.setenv("KG_KERNEL", "full")
        b = g.run_host(X)
    assert b.hits.shape[0] > 0
    for r in (a, again, runs):
        assert r.n_tested == b.n_tested
        assert np.array_equal(r.hits, b.hits)
