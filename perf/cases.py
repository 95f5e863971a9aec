"""The workloads whose speed this framework is judged by.

Every case is one call that a user's program makes through
:mod:`supergwas_b200.api`: the 1-D association test of a batch of packed k-mer
rows against one phenotype (``test``), against many phenotypes at once
(``multi``), or the 2-D test of every pair of k-mers (``pairs``).  Sizes are
those of the repository's own benchmark, tests and fixtures (n = 200 to 5000
samples, r = 2 to 32 principal components, batches from a few thousand to a
hundred million k-mers).

``prepare`` makes what a program has in hand before the call: packed rows on
the device (or on the host, where the program reads them from files), U, y and
a context that holds them.  ``exact`` restates the statistic in plain torch and
numpy, without any code of the package.

Inputs: k-mer frequencies follow Beta(1/2, 1/2), shifted per subpopulation
(F_ST = 0.1) and rounded to 1/256, so that rows absent or present in every
sample occur as in real batches.  A subpopulation is a run of whole 64-sample
words.  U is an orthonormal basis of the intercept, the subpopulation
contrasts and Gaussian columns; y has structure, 20 causal k-mers and noise.
"""
import math

import numpy as np
import torch

from supergwas_b200 import api

F_ST = 0.1
N_CAUSAL = 20
EPS = 1e-12


# ------------------------------------------------------------------ the cases

def _test(name, n, k, m, **opt):
    """One phenotype.  prec: arithmetic form; corr: Pearson gate; missing:
    share of the rows' samples without a phenotype; feed: where the rows are;
    stats: every k-mer's statistics come back, not only the emitted rows."""
    case = dict(name=name, kind="test", n=n, k=k, m=m, prec="split", corr=0.0, log10=6.0, missing=0.0, feed="device",
                stats=False)
    case.update(opt)
    if name is None:
        del case["name"]
    return case


def listed():
    return [
        # The smallest call in earnest: a trial batch in ordinary host memory.
        _test("trial_3k_host", 200, 6, 3000, corr=0.2, feed="pageable"),
        # One batch of a small cohort on the device, at the pipeline's default gate.
        _test("batch_1m_n200", 200, 6, 1_000_000, corr=0.2),
        # Every k-mer's statistics, for a quantile plot of a chromosome's k-mers.
        _test("all_stats_n613", 613, 11, 200_003, stats=True),
        # A mid-size cohort; the rows also hold samples that have no phenotype.
        _test("batch_10m_n700_masked", 700, 9, 10_000_001, corr=0.2, missing=0.12),
        # The benchmark's workload: a large batch resident in device memory.
        _test("batch_100m_n1000", 1000, 17, 100_000_000),
        # A large cohort, one phenotype.
        _test("batch_10m_n2000", 2000, 21, 10_000_000),
        # A very large cohort with many components.
        _test("batch_2m_n5000", 5000, 33, 2_000_000, corr=0.2),
        # The same test in plain double precision.
        _test("fp64_5m_n1000", 1000, 11, 5_000_000, prec="fp64"),
        # What the command line program does with a batch it has read: rows in
        # ordinary host memory, copied and tested chunk by chunk.
        _test("host_1m_n1000", 1000, 17, 1_000_000, corr=0.2, feed="pageable"),
        # Many phenotypes of one cohort, each with its own missing samples.
        dict(name="multi64_4m_n2000", kind="multi", n=2000, k=21, m=4_000_000, phenos=64, corr=0.0, log10=6.0,
             missing=0.3, shards=4),
        # A few phenotypes of a very large cohort.
        dict(name="multi8_1m_n5000", kind="multi", n=5000, k=33, m=1_000_000, phenos=8, corr=0.0, log10=6.0,
             missing=0.3, shards=1),
        # Every pair of a list of k-mers (the interaction scan after the 1-D test).
        dict(name="pairs_20k_n1000", kind="pairs", n=1000, k=17, m=20_000, log10=6.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the ranges above; no more work than the largest listed one."""
    kind = rng.choice(["test"] * 7 + ["fp64"] * 2 + ["host"] * 2 + ["multi"] * 2 + ["pairs"])
    n = _log_int(rng, 150, 5000)
    k = rng.randint(2, max(3, min(33, n // 16)))
    corr = rng.choice([0.0, 0.2])
    missing = rng.choice([0.0, 0.0, rng.uniform(0.02, 0.3)])
    if kind == "multi":
        phenos = _log_int(rng, 3, 64)
        m = _log_int(rng, 20_000, min(4_000_000, 3e12 / (n * k * phenos) + 20_001))
        return dict(kind="multi", n=n, k=k, m=m, phenos=phenos, corr=corr, log10=6.0, missing=rng.uniform(0.0, 0.3),
                    shards=rng.randint(1, 9))
    if kind == "pairs":
        n = min(n, 2000)
        k = min(k, 17)
        return dict(kind="pairs", n=n, k=k, m=_log_int(rng, 500, math.sqrt(2e12 / (n * k))), log10=6.0)
    if kind == "host":
        feed = rng.choice(["pageable", "pinned"])
        m = _log_int(rng, 1000, 1e9 / n)
        return _test(None, n, k, m, corr=corr, missing=missing, feed=feed)
    if kind == "fp64":
        m = _log_int(rng, 5000, 5e10 / (n * k))
        stats = m < 300_000 and rng.random() < 0.3
        return _test(None, n, k, m, prec="fp64", corr=corr, missing=missing, stats=stats)
    m = _log_int(rng, 5000, min(1.5e10 / n, 3e11 / (n * k)))
    stats = m < 300_000 and rng.random() < 0.3
    return _test(None, n, k, m, corr=corr, missing=missing, stats=stats)


def work(case):
    """Each packed row read once, each result written once; the contraction of
    every tested row with the structure columns and the phenotype."""
    n, k, m = case["n"], case["k"], case["m"]
    row = (n + 7) // 8
    bytes_ = m * row
    if case["kind"] == "pairs":
        return {"bytes": bytes_, "flops": m * (m - 1) // 2 * 2 * n * (k + 1)}
    if case["kind"] == "multi":
        return {"bytes": bytes_, "flops": m * 2 * n * (k + 1) * case["phenos"]}
    if case["stats"]:
        bytes_ += m * (1 + 7 * 8)
    return {"bytes": bytes_, "flops": m * 2 * n * (k + 1)}


# ----------------------------------------------------------------- the inputs

def _words(n):
    w = (n + 63) // 64
    return w + (w & 1)


def _subpops(n, k):
    return max(1, min(8, k, (n + 63) // 64))


def _pop_of_word(n, k):
    words, S = (n + 63) // 64, _subpops(n, k)
    return torch.arange(words) * S // words


def _rows(n, k, m, seed, words):
    """m packed rows (int64, m x words) on the GPU, a function of the arguments alone."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(0x5EED ^ (int(seed) * 1_000_003))
    out = torch.zeros((m, words), dtype=torch.int64, device=dev)
    used = (n + 63) // 64
    pop = _pop_of_word(n, k).to(dev)
    S = int(pop.max()) + 1
    tail = n - 64 * (used - 1)
    mask = torch.full((used,), -1, dtype=torch.int64, device=dev)
    if tail < 64:
        mask[-1] = (1 << tail) - 1
    step = max(1, (1 << 24) // used)
    for s in range(0, m, step):
        c = min(step, m - s)
        p = torch.sin(0.5 * math.pi * torch.rand((c, 1), generator=gen, device=dev)) ** 2
        p = p + torch.sqrt(F_ST * p * (1 - p)) * torch.randn((c, S), generator=gen, device=dev)
        p = (p.clamp(0, 1) * 256).round().clamp(0, 255).to(torch.int32)[:, pop]
        # a Bernoulli(p / 256) bit is decided by the first random bit, from the
        # high digit of p down, that differs from p's: digits from the low end,
        # OR where p's digit is 1 and AND where it is 0
        acc = torch.zeros((c, used), dtype=torch.int64, device=dev)
        word = torch.empty_like(acc)
        for digit in range(8):
            word.random_(-(1 << 63), None, generator=gen)
            acc = torch.where((p >> digit & 1).bool(), acc | word, acc & word)
        out[s:s + c, :used] = acc & mask
    return out


def _bits(rows, n):
    """The 0/1 matrix (uint8) of packed rows."""
    by = rows.contiguous().view(torch.uint8).view(rows.shape[0], -1)
    sh = torch.arange(8, dtype=torch.uint8, device=rows.device)
    return ((by.unsqueeze(2) >> sh) & 1).view(rows.shape[0], -1)[:, :n]


def _phenotype(rng, rows, n, k, pos):
    """U (n_ov x k, orthonormal, first column the intercept's) and y over the samples pos."""
    pop = _pop_of_word(n, k).numpy()[np.arange(n) // 64]
    S = _subpops(n, k)
    Z = rng.standard_normal((n, k))
    Z[:, 0] = 1.0
    for s in range(1, S):
        Z[:, s] = (pop == s) + 0.05 * Z[:, s]
    U, _ = np.linalg.qr(Z[pos])
    m = rows.shape[0]
    idx = rng.integers(0, m, min(N_CAUSAL, m))
    X = _bits(rows[torch.as_tensor(idx, device=rows.device)], n).cpu().numpy()[:, pos].astype(np.float64)
    X -= X.mean(axis=1, keepdims=True)
    sd = X.std(axis=1, keepdims=True)
    X /= np.where(sd > 0, sd, 1.0)
    y = X.T @ (rng.standard_normal(idx.size) * 0.35)
    y += Z[pos, 1] * 0.5 + rng.standard_normal(pos.size) + 3.0
    return np.ascontiguousarray(U), y


def _positions(rng, n, missing):
    if missing <= 0:
        return np.arange(n)
    return np.sort(rng.choice(n, size=n - int(missing * n), replace=False))


def _inputs(case, seed):
    """The packed rows on the GPU and, per phenotype, (U, y, sample positions)."""
    n, k, m = case["n"], case["k"], case["m"]
    words = _words(n)
    if case["kind"] == "multi":
        words = max(words, 16)  # the many-phenotype entry point takes rows of 128 bytes and more
    rows = _rows(n, k, m, seed, words)
    rng = np.random.default_rng([int(seed), n, k, m])
    phenos = []
    for _ in range(case.get("phenos", 1)):
        missing = case.get("missing", 0.0)
        if case["kind"] == "multi":
            missing = rng.uniform(0.0, missing)
        pos = _positions(rng, n, missing)
        U, y = _phenotype(rng, rows, n, k, pos)
        phenos.append((U, y, pos))
    return rows, phenos


def _shard_starts(case):
    m, s = case["m"], case["shards"]
    # uneven shards: the i-th starts at m (i / s)^1.5
    return np.array([int(m * (i / s) ** 1.5) for i in range(s)], dtype=np.uint64)


def prepare(case, seed):
    rows, phenos = _inputs(case, seed)
    if case["kind"] == "multi":
        g = api.Kgwas(corr_threshold=case["corr"], log10_thresh=case["log10"])
        g.set_phenotypes(phenos, case["n"])
        torch.cuda.synchronize()
        return {"case": case, "g": g, "rows": rows, "shards": _shard_starts(case)}
    U, y, pos = phenos[0]
    if case["kind"] == "pairs":
        g = api.Kgwas(corr_threshold=0.0, log10_thresh=case["log10"])
        g.set_structure(U, y)
        return {"case": case, "g": g, "host": rows.cpu().numpy().view(np.uint64)}
    g = api.Kgwas(precision=case["prec"], corr_threshold=case["corr"], log10_thresh=case["log10"])
    if pos.size == case["n"]:
        g.set_structure(U, y)
    else:
        g.set_structure(U, y, pos, case["n"])
    state = {"case": case, "g": g}
    if case["feed"] == "device":
        state["rows"] = rows
    else:
        host = rows.cpu()
        if case["feed"] == "pinned":
            host = host.pin_memory()
        state["keep"] = host
        state["host"] = host.numpy().view(np.uint64)
    torch.cuda.synchronize()
    return state


# ---------------------------------------------------------------- one pass

def _room(case):
    """Rows of the table that a pass fills with its emitted rows: a pair list
    runs to a few rows per k-mer, a batch to far fewer."""
    if case["kind"] == "pairs":
        return 1 << (4 * case["m"] - 1).bit_length()
    if case["kind"] == "multi":
        return 65536
    return 256 if case["m"] < 10_000 else 16384


def _table(case, columns):
    """Emitted rows as a program keeps them: one column per field in a table
    with room to spare (doubled when it does not hold them), zeros after the
    last row."""
    room = _room(case)
    while room < len(columns[next(iter(columns))]):
        room *= 2
    out = {}
    for name, values in columns.items():
        out[name] = np.zeros(room, values.dtype)
        out[name][:len(values)] = values
    return out


def _hits(case, hits):
    return {"rows": len(hits), **_table(case, {f: hits[f] for f in hits.dtype.names})}


def run(state):
    case, g = state["case"], state["g"]
    if case["kind"] == "multi":
        rows = state["rows"]
        g.launch_multi_device(rows.data_ptr(), rows.shape[0], rows.shape[1], state["shards"],
                              torch.cuda.current_stream().cuda_stream)
        tested, hits = g.fetch_multi()
        return {"tested": tested.astype(np.int64), **_hits(case, hits)}
    if case["kind"] == "pairs":
        pairs, evaluated = g.run_pairs_host(state["host"])
        return {"evaluated": evaluated, **_hits(case, pairs)}
    stats = case["stats"]
    if case["feed"] == "device":
        rows = state["rows"]
        g.launch_device(rows.data_ptr(), rows.shape[0], rows.shape[1], torch.cuda.current_stream().cuda_stream,
                        stats=stats)
        res = g.fetch(stats=stats)
    else:
        res = g.run_host(state["host"], stats=stats)
    out = {"tested": res.n_tested, **_hits(case, res.hits)}
    if stats:
        out.update({"all_" + f: a for f, a in res.stats.items()})
    return out


# ------------------------------------------------- the same values in 64 bits

class _Model:
    """One phenotype's contraction columns in extended precision.

    A column v is split into a part on a fixed grid, whose sums over samples
    are exact in a double, and the rest; x.v is then good to a rounding."""

    def __init__(self, U, y, pos, n, dev):
        ld = np.longdouble
        U, y = U.astype(ld), y.astype(ld)
        Uy = U.T @ y
        yp = y - U @ Uy                      # x.y - (U'x).(U'y) = x.(y - U U'y)
        yc = y - y.mean()
        self.n, self.k = len(y), U.shape[1]
        self.yyM = float((y * y).sum() - (Uy * Uy).sum())
        self.ynorm = float(np.sqrt((yc * yc).sum()))
        cols = np.concatenate([U, yp[:, None], yc[:, None]], axis=1)
        full = np.zeros((n, cols.shape[1]), dtype=ld)
        full[pos] = cols
        scale = np.exp2(np.ceil(np.log2(np.maximum(np.abs(full).max(axis=0), 1e-300))).astype(np.float64) - 36)
        hi = np.rint((full / scale).astype(np.float64)) * scale
        lo = (full - hi).astype(np.float64)
        self.hi, self.lo = torch.as_tensor(hi, device=dev), torch.as_tensor(lo, device=dev)
        here = np.zeros(n)
        here[pos] = 1.0
        self.here = torch.as_tensor(here, device=dev)

    def statistic(self, c, e, corr):
        """Everything the test reports, from c = popcount and e = [U'x, x.y', x.(y - mean)]."""
        n, k = self.n, self.k
        xxM = c - (e[..., :k] ** 2).sum(-1)
        xyM, xyc = e[..., k], e[..., k + 1]
        inside = (c > 0) & (c < n)
        if self.ynorm < EPS:
            inside = torch.zeros_like(inside)
        xc2 = torch.where(inside, c * (n - c) / n, torch.ones_like(c))
        cor = torch.where(inside, xyc / (torch.sqrt(xc2) * max(self.ynorm, 1e-300)), torch.zeros_like(c))
        tested = inside & ~(cor.abs() < corr)
        return tested, cor, *self.hit(tested, xxM, xyM)

    def hit(self, tested, xxM, xyM):
        ok = tested & (xxM > EPS) & (self.yyM > EPS)
        den = torch.where(ok, xxM * self.yyM, torch.ones_like(xxM))
        r2 = torch.where(ok, xyM * xyM / den, torch.zeros_like(xxM)).clamp(0.0, 1 - 1e-15)
        T = -self.n * torch.log1p(-r2)
        z = torch.sqrt(0.5 * T)
        p = torch.special.erfc(z)
        ml = torch.where(z < 5, -torch.log10(p.clamp_min(1e-300)),
                         (z * z - torch.log(torch.special.erfcx(z))) / math.log(10.0))
        effect = torch.where(ok, xyM / den, torch.zeros_like(xxM))
        zero = torch.zeros_like(xxM)
        return ok, T, p, ml, effect, torch.where(tested, xxM, zero), torch.where(tested, xyM, zero)


def _scan(model, rows, n, corr, log10, keep_all):
    """The 1-D test of every row: tested flags, emitted rows and, with keep_all, all values."""
    m = rows.shape[0]
    tested_all, hits, full = [], [], []
    step = max(1, (1 << 28) // n)
    for s in range(0, m, step):
        x = _bits(rows[s:s + step], n).double()
        c = x @ model.here
        e = x @ model.hi + x @ model.lo
        tested, cor, ok, T, p, ml, effect, xxM, xyM = model.statistic(c, e, corr)
        tested_all.append(tested)
        idx = torch.nonzero(tested & (p <= 10.0 ** -log10)).flatten()
        hits.append([v.cpu().numpy() for v in (idx + s, effect[idx], p[idx], T[idx])])
        if keep_all:
            one, zero = torch.ones_like(p), torch.zeros_like(p)
            full.append([v.cpu().numpy() for v in (T, torch.where(tested, p, one), effect,
                                                   torch.where(tested, ml, zero), xxM, xyM, cor)])
        del x, c, e
    cat = [np.concatenate([h[i] for h in hits]) for i in range(4)]
    every = [np.concatenate([f[i] for f in full]) for i in range(7)] if keep_all else None
    return torch.cat(tested_all), cat, every


def exact(case, seed):
    rows, phenos = _inputs(case, seed)
    n, m, dev = case["n"], case["m"], rows.device
    if case["kind"] == "pairs":
        U, y, pos = phenos[0]
        return _exact_pairs(case, _Model(U, y, pos, n, dev), _bits(rows, n).double())
    if case["kind"] == "multi":
        starts = _shard_starts(case).astype(np.int64)
        edges = torch.as_tensor(np.append(starts, m), device=dev)
        counts = np.zeros((len(starts), len(phenos)), np.int64)
        parts = []
        for p, (U, y, pos) in enumerate(phenos):
            tested, (idx, eff, pv, T), _ = _scan(_Model(U, y, pos, n, dev), rows, n, case["corr"], case["log10"], False)
            run_sum = torch.cat([torch.zeros(1, dtype=torch.int64, device=dev), tested.cumsum(0)])
            counts[:, p] = run_sum[edges].diff().cpu().numpy()
            shard = np.searchsorted(starts, idx, side="right") - 1
            parts.append([idx.astype(np.uint64), np.full(idx.size, p, np.int32), shard.astype(np.int32), eff, pv, T])
        names = ("kmer", "pheno", "shard", "effect", "pval", "chisq")
        cols = {f: np.concatenate([q[i] for q in parts]) for i, f in enumerate(names)}
        return {"tested": counts, "rows": cols["kmer"].size, **_table(case, cols)}
    U, y, pos = phenos[0]
    tested, (idx, eff, pv, T), every = _scan(_Model(U, y, pos, n, dev), rows, n, case["corr"], case["log10"],
                                             case["stats"])
    out = {"tested": int(tested.sum()), "rows": idx.size,
           **_table(case, {"kmer": idx.astype(np.uint64), "effect": eff, "pval": pv, "chisq": T})}
    if case["stats"]:
        names = ("chisq", "pval", "effect", "mlog10p", "xxM", "xyM", "cor")
        out.update({"all_" + f: every[i] for i, f in enumerate(names)})
        out["all_tested"] = tested.cpu().numpy()
    return out


def _exact_pairs(case, model, x):
    """Every pair i < j: the 1-D test of the product column x_i x_j, without the gate."""
    m, k = x.shape[0], model.k
    total, parts = 0, []
    step = max(1, (1 << 24) // m)
    for s in range(0, m, step):
        xi = x[s:s + step]
        xj = x[s:]
        c = xi @ xj.T
        ss = torch.zeros_like(c)
        for j in range(k + 1):
            e = (xi * model.hi[:, j]) @ xj.T + (xi * model.lo[:, j]) @ xj.T
            if j < k:
                ss += e * e
        i_idx = torch.arange(xi.shape[0], device=x.device)[:, None]
        j_idx = torch.arange(xj.shape[0], device=x.device)[None, :]
        valid = (j_idx > i_idx) & (c > 0)
        ok, T, p, _, effect, _, _ = model.hit(valid, c - ss, e)
        total += int(ok.sum())
        sel = torch.nonzero(ok & (p <= 10.0 ** -case["log10"]))
        a, b = sel[:, 0], sel[:, 1]
        parts.append([v.cpu().numpy() for v in (a + s, b + s, effect[a, b], p[a, b], T[a, b])])
    cat = [np.concatenate([q[i] for q in parts]) for i in range(5)]
    cols = {"a": cat[0].astype(np.uint64), "b": cat[1].astype(np.uint64), "effect": cat[2], "pval": cat[3],
            "chisq": cat[4]}
    return {"evaluated": total, "rows": cat[0].size, **_table(case, cols)}
