"""Rows in the span of U (markers of a lineage) stay undecided in the 4-bit
screen whatever their statistic.  With many of them the screen gives up and the
kernel behind it evaluates the launch: the same counts and rows, for this launch
alone.  KG_SCREEN_OPEN moves the point at which it does; the tests of
test_gpu_screen4.py, whose rows are often such, run again with it out of reach."""
import numpy as np
import pytest

import test_gpu_screen4 as S
from supergwas_b200 import api, synth

pytestmark = pytest.mark.gpu
NEVER = str(1 << 24)


def batch(n, k, m, share, rng):
    """m rows, `share` of them subpopulations with 1 % of the samples flipped, and
    a structure that holds the subpopulations."""
    pop, Z = S.structure(n, k, rng)
    x = (rng.random((4096, n)) < rng.random((4096, 1))).astype(np.uint8)
    x[:64] = (pop == np.arange(64)[:, None] % 4) ^ (rng.random((64, n)) < 0.01)
    y = rng.standard_normal(n) + 0.5 * pop
    x[64:80] = (y + rng.standard_normal((16, n))) > 1.0
    mark = rng.random(m) < share
    X = synth.pack_rows(x, max(16, synth.words_per_kmer(n)) if n >= 900 else None)
    X = np.ascontiguousarray(X[np.where(mark, rng.integers(0, 64, m), rng.integers(64, 4096, m))])
    return np.linalg.qr(Z)[0], y, X


# share of markers, KG_SCREEN_OPEN, whether it gives up: none; below and above the limits; nearly from the
# first candidate on; out of reach
CASES = [(0.0, None, False), (0.002, None, False), (0.1, None, True), (1.0, None, True), (0.1, "0", True),
         (0.1, NEVER, False)]


@pytest.mark.parametrize("share,base,over", CASES)
@pytest.mark.parametrize("n,k,m,thr", [(200, 6, 400_001, 0.2), (1000, 17, 150_000, 0.0), (5000, 33, 80_000, 0.0)])
def test_one_phenotype(built, n, k, m, thr, share, base, over, monkeypatch):
    import torch
    rng = np.random.default_rng(n)
    U, y, X = batch(n, k, m, share, rng)
    plain = batch(n, k, 4000, 0.0, np.random.default_rng(1))[2]
    monkeypatch.setenv("KG_DEDUP", "0")
    if base is not None:
        monkeypatch.setenv("KG_SCREEN_OPEN", base)
    with api.Kgwas(corr_threshold=thr, log10_thresh=6.0) as g:
        g.set_structure(U, y)
        a = g.run_host(X)
        assert g.last_screen() == (-1 if over else 1)
        dx = torch.from_numpy(X.view(np.int64)).cuda()
        g.launch_device(dx.data_ptr(), X.shape[0], X.shape[1])
        d = g.fetch()
        assert g.last_screen() == (-1 if over else 1)
        monkeypatch.setenv("KG_CHUNK_MB", "1")
        c = g.run_host(X)
        monkeypatch.delenv("KG_CHUNK_MB")
        monkeypatch.delenv("KG_SCREEN_OPEN", raising=False)
        g.run_host(plain)
        assert g.last_screen() == 1  # the call before left nothing behind
        monkeypatch.setenv("KG_KERNEL", "full")
        b = g.run_host(X)
    assert b.hits.shape[0] > 0 or share == 1.0
    for r in (a, c, d):
        assert r.n_tested == b.n_tested
        assert np.array_equal(r.hits, b.hits)


@pytest.mark.parametrize("share,base,over", CASES)
def test_fp64_form(built, share, base, over, monkeypatch):
    import torch
    n, k, m = 1000, 11, 420_000
    U, y, X = batch(n, k, m, share, np.random.default_rng(n))
    monkeypatch.setenv("KG_DEDUP", "0")
    if base is not None:
        monkeypatch.setenv("KG_SCREEN_OPEN", base)
    with api.Kgwas(precision="fp64", corr_threshold=0.0, log10_thresh=6.0) as g:
        g.set_structure(U, y)
        out = []
        for _ in range(2):
            out.append(g.run_host(X))
            assert g.last_screen() == (-1 if over else 1)
        dx = torch.from_numpy(X.view(np.int64)).cuda()
        g.launch_device(dx.data_ptr(), m, X.shape[1])
        out.append(g.fetch())
        assert g.last_screen() == (-1 if over else 1)
        monkeypatch.setenv("KG_KERNEL", "full")
        b = g.run_host(X)
    for a in out:
        assert a.n_tested == b.n_tested
        assert np.array_equal(a.hits, b.hits)


@pytest.mark.parametrize("share,base,over", CASES)
@pytest.mark.parametrize("n,k", [(900, 12), (2000, 21), (5000, 33)])
def test_many_phenotypes(built, n, k, share, base, over, monkeypatch):
    """Behind the screen: images that share an MMA group, the SM pair and the
    streamed image; host chunks, and device launches that replay a graph."""
    import torch
    rng = np.random.default_rng(n)
    U, y, X = batch(n, k, 30_000, share, rng)
    if base is not None:
        monkeypatch.setenv("KG_SCREEN_OPEN", base)
    phenos = [(U, y + 0.3 * rng.standard_normal(n), np.arange(n)) for _ in range(5)]
    shards = np.array([0, 77, 10_000], dtype=np.uint64)
    monkeypatch.setenv("KG_DEDUP", "0")
    dx = torch.from_numpy(X.view(np.int64)).cuda()
    st = torch.cuda.current_stream().cuda_stream
    out = []
    with api.Kgwas(corr_threshold=0.0, log10_thresh=6.0) as g:
        g.set_phenotypes(phenos, n)
        for _ in range(4):
            g.launch_multi_device(dx.data_ptr(), X.shape[0], X.shape[1], shards, st)
            out.append(g.fetch_multi())
            assert g.last_screen() == (-1 if over else 1)
        monkeypatch.setenv("KG_CHUNK_MB", "1")
        out.append(g.run_multi_host(X, shards))
        monkeypatch.setenv("KG_MP_KERNEL", "mp")
        ref = g.run_multi_host(X, shards)
        assert g.last_screen() == 0
    for tested, hits in out:
        assert np.array_equal(tested, ref[0])
        assert np.array_equal(hits, ref[1])


@pytest.mark.parametrize("share,base,over", CASES[1:])
def test_pairs(built, share, base, over, monkeypatch):
    n, k, m = 1000, 17, 1500
    U, y, X = batch(n, k, m, share, np.random.default_rng(n))
    if base is not None:
        monkeypatch.setenv("KG_SCREEN_OPEN", base)
    with api.Kgwas(corr_threshold=0.0, log10_thresh=6.0) as g:
        g.set_structure(U, y)
        for r0, r1 in ((0, m), (m // 3, m // 3 + 200)):
            a, ea = g.run_pairs_host(X, r0, r1)
            if share in (0.002, 1.0):
                assert (g.last_screen() < 0) == over
            monkeypatch.setenv("KG_KERNEL", "full")
            b, eb = g.run_pairs_host(X, r0, r1)
            monkeypatch.delenv("KG_KERNEL")
            assert ea == eb
            assert np.array_equal(a, b)


@pytest.mark.parametrize("n,k,m", S.SHAPES, ids=lambda v: str(v))
@pytest.mark.parametrize("thr,lt", [(0.0, 6.0), (0.2, 4.0), (1e-5, 9.0)])
def test_awkward_rows_on_the_screen(built, n, k, m, thr, lt, monkeypatch):
    monkeypatch.setenv("KG_SCREEN_OPEN", NEVER)
    S.test_same_rows_as_full_kernel(built, n, k, m, thr, lt, monkeypatch)


@pytest.mark.parametrize("tail", ["y", "U", "both", "scale"])
@pytest.mark.parametrize("thr", [0.0, 0.1])
def test_heavy_tails_on_the_screen(built, tail, thr, monkeypatch):
    monkeypatch.setenv("KG_SCREEN_OPEN", NEVER)
    S.test_heavy_tails_and_missing_samples(built, tail, thr, monkeypatch)


@pytest.mark.parametrize("thr,lt", [(0.0, 6.0), (0.2, 4.0)])
@pytest.mark.parametrize("n,ks,np_", [(900, (12, 15), 5), (2000, (21, 3), 7), (1030, (5, 6), 17), (5000, (33, 30), 3),
                                      (300, (2, 3), 8)], ids=lambda v: str(v))
def test_many_phenotypes_on_the_screen(built, n, ks, np_, thr, lt, monkeypatch):
    monkeypatch.setenv("KG_SCREEN_OPEN", NEVER)
    S.test_many_phenotypes(built, n, ks, np_, thr, lt, monkeypatch)


@pytest.mark.parametrize("n,k,m", [(1000, 17, 700), (300, 4, 1501), (2000, 21, 400), (1024, 9, 130)],
                         ids=lambda v: str(v))
@pytest.mark.parametrize("thr", [0.0, 0.2])
def test_pairs_on_the_screen(built, n, k, m, thr, monkeypatch):
    monkeypatch.setenv("KG_SCREEN_OPEN", NEVER)
    S.test_pairs(built, n, k, m, thr, monkeypatch)


def test_longer_candidate_list_between_graph_replays(built):
    """A large launch of one phenotype makes the shared candidate list longer; the
    captured launches of many phenotypes take the new one."""
    import torch
    rng = np.random.default_rng(2)
    U, y, X = batch(900, 12, 4000, 0.0, rng)
    n = 60
    big = torch.empty((70_000_000, 2), dtype=torch.int64, device="cuda").random_()
    big[:, 0] &= (1 << n) - 1
    big[:, 1] = 0
    st = torch.cuda.current_stream().cuda_stream
    dx = torch.from_numpy(X.view(np.int64)).cuda()
    out = []
    with api.Kgwas(corr_threshold=0.0, log10_thresh=6.0) as g:
        g.set_phenotypes([(U, y, np.arange(900))] * 3, 900)
        g.set_structure(np.full((n, 1), n ** -0.5), rng.standard_normal(n))
        for i in range(6):
            g.launch_multi_device(dx.data_ptr(), X.shape[0], X.shape[1], None, st)
            out.append(g.fetch_multi())
            if i == 3:
                g.launch_device(big.data_ptr(), big.shape[0], 2, st)
                g.fetch()
                assert g.last_screen() == 1
    for tested, hits in out[1:]:
        assert np.array_equal(tested, out[0][0]) and np.array_equal(hits, out[0][1])


@pytest.mark.parametrize("prec,m", [("split", 150_000), ("fp64", 420_000), ("many", 30_000)])
@pytest.mark.parametrize("share", [0.0, 0.3])
def test_rows_overwritten_behind_the_launch(built, prec, m, share, monkeypatch):
    """A launch has read its rows when the stream is past it, whether the screen
    gives up or not: the next rows may go to the same buffer before the fetch."""
    import torch
    n, k = (1000, 11) if prec == "fp64" else (1000, 17)
    U, y, X = batch(n, k, m, share, np.random.default_rng(m))
    rows = torch.from_numpy(X.view(np.int64)).cuda()
    dx = rows.clone()
    stream = torch.cuda.Stream()  # 0 would be the context's own stream
    st = stream.cuda_stream
    stream.wait_stream(torch.cuda.current_stream())
    form = "split" if prec == "many" else prec
    with torch.cuda.stream(stream), api.Kgwas(precision=form, corr_threshold=0.0, log10_thresh=6.0) as g:
        if prec == "many":
            g.set_phenotypes([(U, y + 0.1 * p, np.arange(n)) for p in range(3)], n)
            ref = g.run_multi_host(X)
            for _ in range(3):
                dx.copy_(rows)
                g.launch_multi_device(dx.data_ptr(), m, X.shape[1], None, st)
                dx.zero_()
                tested, hits = g.fetch_multi()
                assert np.array_equal(tested, ref[0]) and np.array_equal(hits, ref[1])
        else:
            g.set_structure(U, y)
            g.launch_device(dx.data_ptr(), m, X.shape[1], st)
            dx.zero_()
            r = g.fetch()
            monkeypatch.setenv("KG_KERNEL", "full")
            ref = g.run_host(X)
            assert r.n_tested == ref.n_tested and np.array_equal(r.hits, ref.hits)
        assert ref[1].shape[0] > 0 if prec == "many" else ref.hits.shape[0] > 0
