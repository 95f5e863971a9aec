"""Which calls the 4-bit screen takes.  The tests that compare it with the
kernels that evaluate every k-mer (test_gpu_screen4.py) hold whether it runs or
not: here it is asked for, shape by shape."""
import numpy as np
import pytest

from supergwas_b200 import api, synth
from test_gpu_screen4 import SHAPES, structure

pytestmark = pytest.mark.gpu


def rows_of(n, m, rng):
    X = synth.pack_rows((rng.random((2048, n)) < rng.random((2048, 1))).astype(np.uint8))
    return np.ascontiguousarray(X[np.arange(m) % X.shape[0]])


# work that the screen would not save its cost on (3e9 k-mers x samples x limb columns, above 4096 k-mers)
SMALL = {(200, 6, 60_001), (640, 11, 20_000), (1000, 17, 40_000)}


@pytest.mark.parametrize("n,k,m", SHAPES, ids=lambda v: str(v))
@pytest.mark.parametrize("thr,lt", [(0.0, 6.0), (0.2, 4.0), (1e-5, 9.0)])
def test_one_phenotype(built, n, k, m, thr, lt, monkeypatch):
    rng = np.random.default_rng(n + k + m)
    pop, Z = structure(n, k, rng)
    y = rng.standard_normal(n) + 0.5 * pop + 2.0
    X = rows_of(n, m, rng)
    monkeypatch.setenv("KG_DEDUP", "0")
    with api.Kgwas(corr_threshold=thr, log10_thresh=lt) as g:
        g.set_structure(np.linalg.qr(Z)[0], y)
        g.run_host(X)
        assert g.last_screen() == ((n, k, m) not in SMALL)
        monkeypatch.setenv("KG_SCREEN_OPEN", str(1 << 24))
        g.run_host(X)
        assert g.last_screen() == 1
        monkeypatch.delenv("KG_SCREEN_OPEN")
        g.run_host(X[:1], stats=True)
        assert g.last_screen() == 0
        monkeypatch.setenv("KG_KERNEL", "full")
        g.run_host(X)
        assert g.last_screen() == 0


@pytest.mark.parametrize("tail,limbs", [("y", 1), ("U", 2), ("scale", 0), ("threshold", 0), ("missing", 1)])
def test_structures_that_need_more_or_are_refused(built, tail, limbs):
    n, k = 1200, 12
    rng = np.random.default_rng(len(tail))
    pop, Z = structure(n, k, rng)
    if tail == "U":
        Z[:, 5:] = rng.standard_cauchy((n, k - 5))
    y = rng.standard_cauchy(n) if tail == "y" else rng.standard_normal(n) + 0.5 * pop
    keep = np.arange(n) if tail != "missing" else np.sort(rng.choice(n, n - n // 7, replace=False))
    U = np.linalg.qr(Z[keep])[0] * (1.5 if tail == "scale" else 1.0)
    with api.Kgwas(corr_threshold=0.0, log10_thresh=2.0 if tail == "threshold" else 6.0) as g:
        g.set_structure(U, y[keep], keep, n)
        g.run_host(rows_of(n, 3000, rng))
        assert g.last_screen() == limbs


@pytest.mark.parametrize("n,k,m", [(1000, 17, 700), (300, 4, 1501), (2000, 21, 400), (1024, 9, 130)],
                         ids=lambda v: str(v))
@pytest.mark.parametrize("thr", [0.0, 0.2])
def test_pairs(built, n, k, m, thr, monkeypatch):
    rng = np.random.default_rng(n + m)
    pop, Z = structure(n, k, rng)
    y = rng.standard_normal(n) + 0.5 * pop
    X = rows_of(n, m, rng)
    with api.Kgwas(corr_threshold=thr, log10_thresh=4.0) as g:
        g.set_structure(np.linalg.qr(Z)[0], y)
        g.run_pairs_host(X, 0, 40)
        assert g.last_screen() == 1
        monkeypatch.setenv("KG_KERNEL", "full")
        g.run_pairs_host(X, 0, 40)
        assert g.last_screen() == 0


@pytest.mark.parametrize("n,k,m,screened", [(1000, 11, 420_001, True), (300, 12, 900_001, True),
                                            (2100, 21, 100_001, True), (1000, 11, 20_000, False)],
                         ids=lambda v: str(v))
def test_fp64_form(built, n, k, m, screened, monkeypatch):
    rng = np.random.default_rng(n + m)
    pop, Z = structure(n, k, rng)
    y = rng.standard_normal(n) + 0.5 * pop
    monkeypatch.setenv("KG_DEDUP", "0")
    with api.Kgwas(precision="fp64", corr_threshold=0.0, log10_thresh=6.0) as g:
        g.set_structure(np.linalg.qr(Z)[0], y)
        X = synth.pack_rows((rng.random((2048, n)) < rng.random((2048, 1))).astype(np.uint8))
        g.run_host(np.ascontiguousarray(X[np.arange(m) % 2048]))
        assert (g.last_screen() > 0) == screened


def test_many_phenotypes(built, monkeypatch):
    n, k = 900, 12
    rng = np.random.default_rng(1)
    pop, Z = structure(n, k, rng)
    y = rng.standard_normal(n) + 0.5 * pop
    U = np.linalg.qr(Z)[0]
    X = rows_of(n, 3000, rng)
    with api.Kgwas(corr_threshold=0.0, log10_thresh=6.0) as g:
        g.set_phenotypes([(U, y, np.arange(n))] * 3, n)
        g.run_multi_host(X)
        assert g.last_screen() == 1
        g.set_phenotypes([(U, y, np.arange(n)), (1.5 * U, y, np.arange(n))], n)  # one without: none
        g.run_multi_host(X)
        assert g.last_screen() == 0
