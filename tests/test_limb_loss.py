"""What the int8 limbs leave out of a row's sums, and the tests that are left
undecided, or unrefined, on account of it.  Columns that mark single samples
round nearly every value the same way, so a row that misses a few samples meets
the sum of n roundings: at n = 24000, 20 such columns, 19 % of xxM."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from oracle import oracle as O
from supergwas_b200 import api, build, synth

HERE = os.path.dirname(os.path.abspath(__file__))


def marked_samples(n, marks):
    """The intercept and `marks` columns that each mark one sample, with sums of
    exactly zero (multiples of 2^-40), so that the columns are tested as they are."""
    Z = np.full((n, marks), -1.0 / n)
    Z[np.arange(marks), np.arange(marks)] += 1.0
    U = np.rint(np.linalg.qr(Z)[0] * 2.0 ** 40)
    U[np.arange(marks), np.arange(marks)] -= U.sum(axis=0)
    return np.column_stack([np.full(n, 1.0 / np.sqrt(n)), U * 2.0 ** -40])


def held(d, nl):
    """Column d as its limbs hold it."""
    s = np.frexp(127.0 * 2.0 ** (8 * (nl - 1) - 1) / np.abs(d).max())[1] - 1
    return np.rint(np.ldexp(d, s)) * 2.0 ** -float(s)


@pytest.fixture(scope="module")
def constants():
    out = os.path.join(HERE, "native", "_build", "libscreen_check.so")
    src = [os.path.join(HERE, "native", "screen_check.cpp"), os.path.join(build.CSRC, "prep.cpp")]
    os.makedirs(os.path.dirname(out), exist_ok=True)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-D__host__=", "-D__device__=", "-o", out,
                    *src], check=True)
    fn = ctypes.CDLL(out).screen_constants
    vp = ctypes.c_void_p
    fn.argtypes = [vp, ctypes.c_int, ctypes.c_int, vp, ctypes.c_double, ctypes.c_double, vp, vp, vp, vp]

    def call(U, y, chi_cut):
        U, y = np.asfortranarray(U), np.ascontiguousarray(y)
        loss, need, on = np.zeros(2), ctypes.c_double(), ctypes.c_int()
        d = np.zeros((U.shape[1] + 1, U.shape[0]))
        cut, ref = (-np.expm1(-t / U.shape[0]) for t in (chi_cut, 12.0))
        assert fn(U.ctypes.data, *U.shape, y.ctypes.data, cut, ref, loss.ctypes.data, ctypes.byref(need),
                  ctypes.byref(on), d.ctypes.data) == 0
        return loss, need.value / cut, bool(on.value), d
    return call


@pytest.mark.parametrize("n,marks,covered", [(200, 5, True), (2000, 3, True), (24000, 20, False), (40000, 10, False)])
def test_bound_holds_and_decides(constants, n, marks, covered):
    rng = np.random.default_rng(n)
    U, y = marked_samples(n, marks), rng.standard_normal(n)
    loss, need, on, d = constants(U, y, 23.93)
    assert need == pytest.approx(0.9 if covered else 0.0)
    assert on  # undecided by its own rounding in no case
    R = np.stack([d[j] - held(d[j], 3) for j in range(1, marks + 1)], axis=1)
    ry = d[marks + 1] - held(d[marks + 1], 5)
    worst = worst_y = 0.0
    for x in (np.r_[np.zeros(marks + 1), np.ones(n - marks - 1)], np.arange(n) > 0, rng.random(n) < 0.3,
              R[:, 0] > 0, np.arange(n) < marks + 1):
        c = x.sum()
        if not 0 < c < n:
            continue
        worst = max(worst, np.linalg.norm(x @ R) / np.sqrt(c * (n - c) / n))
        worst_y = max(worst_y, abs(x @ ry) / np.sqrt(c * (n - c) / n))
    assert 0.02 * loss[0] < worst <= loss[0] and worst_y <= loss[1]
    # the share of xxM that this may move, at the smallest xxM that is trusted
    assert ((2 * loss[0] + loss[0] ** 2) / 0.02 < 0.1) == covered


def test_ordinary_structures_keep_the_screen(constants):
    rng = np.random.default_rng(3)
    for n, k in ((150, 2), (1000, 17), (5000, 33), (12000, 21)):
        Z = rng.standard_normal((n, k))
        Z[:, 0] = 1.0
        for scale in (1.0, 1e-9, 1e9):
            _, need, on, _ = constants(np.linalg.qr(Z)[0], scale * (rng.standard_normal(n) + 3.0), 23.93)
            assert need == pytest.approx(0.9) and on


@pytest.mark.gpu
@pytest.mark.parametrize("many", [False, True])
def test_rows_near_the_cut_are_emitted(built, many, monkeypatch):
    """Rows that miss every marked sample and one more: xxM is 5 % of
    c (n - c) / n and 19 % too high in the limbs, and chi-square runs from below
    the emit cut to well above it."""
    n, marks, m = 24_000, 20, 400
    rng = np.random.default_rng(11)
    U, y = marked_samples(n, marks), rng.standard_normal(n)
    y[marks:marks + m] = np.linspace(5.5, 7.5, m) * y.std()
    x = np.ones((m, n), dtype=np.uint8)
    x[:, :marks] = 0
    x[np.arange(m), marks + np.arange(m)] = 0
    X = synth.pack_rows(x)
    o = O.cols_stats(X, n, U, y, 0.0)
    want = np.nonzero(o["pval"] <= 1e-6)[0]
    chi = o["chisq"][want]
    assert (chi < 24.5).sum() > 5 and (chi > 28).sum() > 5 and want.size < m - 5
    monkeypatch.setenv("KG_DEDUP", "0")
    with api.Kgwas(corr_threshold=0.0, log10_thresh=6.0) as g:
        if many:
            g.set_phenotypes([(U, y, np.arange(n))] * 2, n)
            tested, hits = g.run_multi_host(X)
            assert np.all(tested == o["n_tested"])
            hits = hits[hits["pheno"] == 1]
        else:
            g.set_structure(U, y)
            r = g.run_host(X)
            assert r.n_tested == o["n_tested"]
            hits = r.hits
    near = np.abs(o["pval"] / 1e-6 - 1.0) < 1e-6
    assert not near[want].any()
    assert np.array_equal(hits["kmer"].astype(np.int64), want)
