"""The tensor-memory kernel on rows shorter than one 128-byte TMA box row and on
limb images that nearly fill shared memory: bit for bit the smem-A kernel's
statistics (both sum the same integers and evaluate the same expressions).
Without per-k-mer outputs the tensor-memory kernel decides most k-mers in
single precision; counts and rows must stay the same."""
import numpy as np
import pytest

from supergwas_b200 import api, synth

pytestmark = pytest.mark.gpu

# (samples, k-mers, principal components): row widths of 16, 32, ..., 112
# bytes, tiles of 1, 127, 128 and 129 k-mers and many tiles per SM, images of
# 128 KB and more
SHAPES = [(1, 50, 0), (64, 127, 3), (128, 128, 4), (129, 129, 5), (250, 60_001, 5), (300, 2049, 12), (500, 1, 6),
          (640, 20_000, 10), (700, 777, 32), (896, 3000, 16), (2000, 3001, 20), (1700, 40_000, 24), (2300, 1500, 22),
          (4000, 2000, 10)]


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


def awkward_rows(n, m, pop, y, rng):
    """Rows around every decision: random ones of all frequencies, single and
    all-but-one samples, subpopulation indicators and their complements with a
    few samples flipped (nearly in the span of U), and rows that follow y."""
    p = np.sin(0.5 * np.pi * rng.random((m, 1))) ** 2
    x = (rng.random((m, n)) < p).astype(np.uint8)
    for i in range(0, m, 8):
        x[i] = 0
        x[i, rng.integers(0, n, 1 + i % 3)] = 1
    for i in range(1, m, 8):
        x[i] = 1
        x[i, rng.integers(0, n, 1 + i % 3)] = 0
    for i in range(2, m, 8):
        x[i] = pop == i // 8 % (pop.max() + 1)
        x[i, rng.integers(0, n, i // 8 % 4)] ^= 1
    for i in range(3, m, 8):
        x[i] = (y + rng.standard_normal(n) * rng.choice([0.5, 1.0, 2.0, 4.0]) * y.std()) > np.quantile(y, rng.random())
    for i in range(4, m, 64):
        x[i] = i & 1
    return x


@pytest.mark.parametrize("lt", [1.0, 4.0, 6.0, 9.0])
@pytest.mark.parametrize("thr", [0.0, 1e-5, 0.2])
@pytest.mark.parametrize("n,k,scale", [(190, 6, 1.0), (1000, 17, 1e-9), (1000, 17, 1e-3), (1500, 30, 1e12)])
def test_screened_rows_equal_smem_kernel(built, n, k, scale, thr, lt, monkeypatch):
    rng = np.random.default_rng(n + k)
    pop = np.arange(n) * 5 // n
    Z = rng.standard_normal((n, k))
    Z[:, 0] = 1.0
    for s in range(1, min(5, k)):
        Z[:, s] = pop == s
    U = np.linalg.qr(Z)[0]
    y = (rng.standard_normal(n) + 0.5 * pop + 2.0) * scale
    X = synth.pack_rows(awkward_rows(n, 20_000, pop, y, rng))
    out = {}
    for kern in ("ts", "ss"):
        monkeypatch.setenv("KG_KERNEL", kern)
        with api.Kgwas(corr_threshold=thr, log10_thresh=lt) as g:
            yyM = g.set_structure(U, y)
            out[kern] = g.run_host(X)
    assert out["ts"].hits.shape[0] > 0 or yyM <= 1e-12  # no row has a p-value below 1 then (src/kgwas.cpp:46)
    assert out["ts"].n_tested == out["ss"].n_tested
    assert np.array_equal(out["ts"].hits, out["ss"].hits)
