"""The waits of the kernels that test_gpu_timeout.py does not reach run out in
the same way, without a fault: the 4-bit screen for one phenotype and for many,
the streamed image, the FP64 form with and without the screen.  The next call on
the same context is right."""
import time

import numpy as np
import pytest

from supergwas_b200 import api
from test_gpu_screen_gives_up import batch

pytestmark = pytest.mark.gpu
ERR_TIMEOUT = 5  # include/kgwas_cuda.h

# samples, U columns, k-mers, precision, -log10 p, kg_last_kernel, limbs of the screen
CASES = {"screen": (1000, 17, 100_000, "split", 6.0, "ts", 1),
         "screen, short rows": (200, 6, 400_000, "split", 6.0, "ts", 1),
         "screen, long rows": (5000, 33, 40_000, "split", 6.0, "ts", 1),
         "streamed image": (5000, 33, 40_000, "split", 2.0, "tb", 0),
         "fp64": (1000, 11, 100_000, "fp64", 6.0, "fp64", 0),
         "fp64 behind the screen": (1000, 11, 420_000, "fp64", 6.0, "fp64", 1)}


@pytest.mark.parametrize("case", list(CASES))
def test_one_phenotype(built, case, monkeypatch):
    import torch
    n, k, m, prec, lt, kernel, limbs = CASES[case]
    U, y, X = batch(n, k, m, 0.0, np.random.default_rng(n))
    dx = torch.from_numpy(X.view(np.int64)).cuda()
    st = torch.cuda.current_stream().cuda_stream
    with api.Kgwas(precision=prec, corr_threshold=0.0, log10_thresh=lt) as g:
        g.set_structure(U, y)
        g.set_wait_limit(1_000_000)  # 1 ms
        g.inject_stall(1)            # each CTA loads one box of rows, then stops
        t0 = time.perf_counter()
        g.launch_device(dx.data_ptr(), m, X.shape[1], st)
        with pytest.raises(api.KgError) as ei:
            g.fetch()
        assert ei.value.code == ERR_TIMEOUT and time.perf_counter() - t0 < 1.5
        assert g.last_kernel() == kernel and g.last_screen() == limbs
        out = []
        for limit in (1_000_000, 0):
            g.set_wait_limit(limit)
            g.launch_device(dx.data_ptr(), m, X.shape[1], st)
            out.append(g.fetch())
        monkeypatch.setenv("KG_KERNEL", "full")
        out.append(g.run_host(X))
    for r in out[:2]:
        assert r.n_tested == out[2].n_tested and np.array_equal(r.hits, out[2].hits)


@pytest.mark.parametrize("n,k,np_", [(1000, 17, 2), (1000, 17, 9)])  # one group and several
def test_many_phenotypes(built, n, k, np_, monkeypatch):
    import torch
    rng = np.random.default_rng(np_)
    U, y, X = batch(n, k, 100_000, 0.0, rng)
    dx = torch.from_numpy(X.view(np.int64)).cuda()
    st = torch.cuda.current_stream().cuda_stream
    with api.Kgwas(corr_threshold=0.0, log10_thresh=6.0) as g:
        g.set_phenotypes([(U, y + rng.standard_normal(n), np.arange(n)) for _ in range(np_)], n)
        launch = lambda: g.launch_multi_device(dx.data_ptr(), X.shape[0], X.shape[1], None, st)
        for _ in range(3):  # the third launch replays a graph
            launch()
            ref = g.fetch_multi()
        g.set_wait_limit(1_000_000)
        g.inject_stall(1)
        t0 = time.perf_counter()
        launch()
        with pytest.raises(api.KgError) as ei:
            g.fetch_multi()
        assert ei.value.code == ERR_TIMEOUT and time.perf_counter() - t0 < 1.5
        assert g.multi_shape()["kernel"] == "4-bit screen (fs)"
        for _ in range(3):
            launch()
            tested, hits = g.fetch_multi()
            assert np.array_equal(tested, ref[0]) and np.array_equal(hits, ref[1])
