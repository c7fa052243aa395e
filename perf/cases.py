"""What a user of this framework has it do, as cases that can be timed.

Every case is one call (or one pass of calls) of the public API on inputs made from a seed:

  counts   one or several query files, in host memory, against a resident database: the count matrix and
           the overlap base pairs (Context.query_counts)
  batch    a set of query files of uneven sizes in device memory, in one call (Context.query_batch_device)
  pairs    the list of overlapping pairs of one query file (Context.query_pairs)
  moments  the sliding-window moments of one source on one chromosome (Moments.build)
  pvalues  the length groups and p-values of a batch of query files (Moments.batch_pvalues_device)

Databases are the two that the benchmark names: 64 files of 50,000 intervals each, and 1,000 files with
Zipf(1.1) sizes and 5% broad intervals, both on 24 chromosomes of 50M-250M bp with log-normal lengths
(median 500 bp).  listed() spans them from a file of a thousand intervals (latency) to a file of 1e5
against 2e9 database intervals; draw() gives more of the same ranges.
"""
import math

import numpy as np
import torch

import riggle_b200 as rg
from riggle_b200 import api

DEV = "cuda:0"
CHROMS = 24


def listed():
    return [
        # an interactive query: a short BED file against a small panel of tracks; latency only
        dict(name="file_1k_db64", kind="counts", db_files=64, db_intervals=3_200_000, queries=1_000, rows=1, overlap=True),
        # the plain small configuration of the benchmark
        dict(name="file_10k_db64", kind="counts", db_files=64, db_intervals=3_200_000, queries=10_000, rows=1, overlap=True),
        # the plain configuration at GPU scale: one file of 1e5 intervals against 2e9 database intervals
        dict(name="file_100k_db2e9", kind="counts", db_files=1000, db_intervals=2_000_000_000, queries=100_000, rows=1,
             overlap=True),
        # a large file (dense peak calls) against a mid-size database, counts alone
        dict(name="file_1m_db3e8_counts", kind="counts", db_files=1000, db_intervals=300_000_000, queries=1_000_000, rows=1,
             overlap=False),
        # a folder of BED files queried in one host call: 37 rows whose intervals share the chromosomes' blocks
        dict(name="rows_37_db64", kind="counts", db_files=64, db_intervals=3_200_000, queries=101_750, rows=37, overlap=True),
        # many query files of 1e2..1e6 intervals, sorted as BED files are, replayed as a graph
        dict(name="batch_256_db64", kind="batch", db_files=64, db_intervals=3_200_000, files=256, largest=1_000_000,
             ordered=True, graph=True),
        # a smaller set of files in any order against a large database, launched directly
        dict(name="batch_48_db2e8", kind="batch", db_files=1000, db_intervals=200_000_000, files=48, largest=1_000_000,
             ordered=False, graph=False),
        # the intervals mode: every overlapping pair of a file, with its base pairs
        dict(name="pairs_100k_db64", kind="pairs", db_files=64, db_intervals=3_200_000, queries=100_000, rows=1),
        # moments of a small source on a short chromosome (chr21 at 100 bp bins): the most frequent build
        dict(name="moments_chr21", kind="moments", bins=467_100, bin=100, intervals=2_000, precision="fp64"),
        # a large source on the longest chromosome (chr1 at 100 bp bins)
        dict(name="moments_chr1", kind="moments", bins=2_489_563, bin=100, intervals=400_000, precision="fp64"),
        # the compensated single-precision path at 64 bp bins
        dict(name="moments_2m_fp32c", kind="moments", bins=2_097_152, bin=64, intervals=9_000, precision="fp32c"),
        # the statistics stage of a batch: p-values of 128 files against 500 sources
        dict(name="pvalues_128x500", kind="pvalues", files=128, largest=200_000, sources=500),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_db(rng, largest):
    if rng.random() < 0.5:
        f = rng.randint(16, 128)
        return dict(db_files=f, db_intervals=f * rng.randint(20_000, 80_000))
    return dict(db_files=1000, db_intervals=_log_uniform(rng, 100_000_000, largest))


def draw(rng):
    kind = rng.choice(["counts", "counts", "counts", "batch", "batch", "pairs", "moments", "moments", "pvalues"])
    if kind == "counts":
        rows = rng.choice([1, 1, rng.randint(2, 64)])
        c = dict(kind=kind, **_draw_db(rng, 1_000_000_000))
        c.update(queries=_log_uniform(rng, 1_000, 1_000_000 if rows == 1 else 200_000), rows=rows, overlap=rng.random() < 0.75)
        return c
    if kind == "batch":
        return dict(kind=kind, **_draw_db(rng, 200_000_000), files=_log_uniform(rng, 4, 48),
                    largest=_log_uniform(rng, 50_000, 1_000_000), ordered=rng.random() < 0.5, graph=rng.random() < 0.5)
    if kind == "pairs":
        f = rng.randint(16, 128)
        return dict(kind=kind, db_files=f, db_intervals=f * rng.randint(20_000, 50_000),
                    queries=_log_uniform(rng, 1_000, 100_000), rows=rng.choice([1, rng.randint(2, 64)]))
    if kind == "moments":
        size = rng.choice([64, 100])
        return dict(kind=kind, bins=_log_uniform(rng, 400_000, 2_480_000), bin=size, intervals=_log_uniform(rng, 1_000, 400_000),
                    precision=rng.choice(["fp64", "fp64", "fp32c"]))
    return dict(kind=kind, files=rng.randint(8, 128), largest=_log_uniform(rng, 20_000, 200_000), sources=rng.randint(64, 500))


# ---- inputs ---------------------------------------------------------------------------------------
def _index(case, seed):
    cl = rg.synth_chrom_lengths(1, CHROMS)
    if case["db_files"] == 1000:
        sizes = rg.synth_zipf_sizes(1000, 1.1, 1000, 10_000_000, case["db_intervals"])
        return cl, rg.Index.synth(rg.SynthSpec(2 * seed + 1, cl, sizes, broad_fraction=0.05))
    sizes = np.full(case["db_files"], case["db_intervals"] // case["db_files"], np.uint64)
    return cl, rg.Index.synth(rg.SynthSpec(2 * seed + 1, cl, sizes))


def _lengths(rng, n, most):
    return np.clip(np.exp(rng.normal(math.log(500.0), 1.0, n)), 20, min(100_000, most)).astype(np.int64)


def _host_file(cl, seed, queries, rows):
    """{chromosome: uint32[n, 3] (start, end, row)}, sorted by (row, start) as files read one after another are."""
    rng = np.random.default_rng([seed, 11])
    share = cl.astype(np.float64) / float(cl.sum())
    out = {}
    for c, n in enumerate(rng.multinomial(queries, share)):
        if n:
            ln = _lengths(rng, n, int(cl[c]) - 1)
            st = (rng.random(n) * (int(cl[c]) - ln)).astype(np.int64)
            row = rng.integers(0, rows, n)
            o = np.lexsort((st, row))
            out[c] = np.ascontiguousarray(np.stack([st, st + ln, row], 1)[o].astype(np.uint32))
    return out


def _file_sizes(case, seed):
    rng = np.random.default_rng([seed, 12])
    return np.exp(rng.uniform(math.log(100.0), math.log(case["largest"]), case["files"])).astype(np.uint64)


def _device_files(case, seed, cl):
    """A file-major batch in device memory: (DeviceBatch, its int32[n, 3] tensor)."""
    spec = rg.SynthSpec(2 * seed + 2, cl, _file_sizes(case, seed), hotspot_fraction=0.1, num_hotspots=8)
    off, shards, rows = rg.synth_batch_layout(spec)
    iv = torch.empty((int(off[-1]), 3), dtype=torch.int32, device=DEV)
    rg.synth_batch_device(spec, off, iv.data_ptr())
    torch.cuda.synchronize()
    if case.get("ordered"):
        cnt = torch.from_numpy(np.diff(off.astype(np.int64))).to(DEV)
        blk = torch.repeat_interleave(torch.arange(len(cnt), device=DEV), cnt)
        o = torch.sort((blk << 32) | iv[:, 0].to(torch.int64)).indices
        iv = iv[o].contiguous()
        torch.cuda.synchronize()
    return rg.DeviceBatch(case["files"], shards, off, iv.data_ptr(), rows), iv


def _moment_intervals(case, seed):
    """One source's intervals on one chromosome, in file order (sorted by start)."""
    rng = np.random.default_rng([seed, 13])
    length = case["bins"] * case["bin"] - 1
    ln = _lengths(rng, case["intervals"], length)
    st = np.sort((rng.random(case["intervals"]) * (length - ln)).astype(np.int64))
    return np.stack([st, st + ln, np.zeros_like(st)], 1).astype(np.uint32)


PV_BIN = 100


def _pvalue_inputs(case, seed):
    """The statistics stage's inputs: chromosome bin counts, per-source coverage and dispersion that set the moment
    tables, the observed overlaps, and the files (through the caller)."""
    cl = rg.synth_chrom_lengths(1, CHROMS)
    bins = (cl.astype(np.int64) // PV_BIN + 1).astype(np.uint64)
    rng = np.random.default_rng([seed, 14])
    cover = np.exp(rng.uniform(math.log(1e-3), math.log(0.3), case["sources"]))
    spread = np.exp(rng.uniform(math.log(0.3), math.log(30.0), case["sources"]))
    noise = np.exp(rng.normal(0.0, 0.05, (case["files"], case["sources"])))
    empty = rng.random((case["files"], case["sources"])) < 0.05
    return cl, bins, cover, spread, noise, empty


def _moment_grid(n):
    """The L grid of a moment table: 1..100, then factors of 1.01 rounded up, below n."""
    ls = list(range(1, min(100, n - 1) + 1))
    x = 100.0
    while True:
        x *= 1.01
        v = math.ceil(x)
        if v > n - 1:
            return np.array(ls, np.int64)
        if v > ls[-1]:
            ls.append(v)


def _observed(case, seed, batch, iv):
    """(counts, base pairs) near what the moment tables predict, so that the tails are of every size."""
    _, _, cover, _, noise, empty = _pvalue_inputs(case, seed)
    ln = (iv[:, 1] - iv[:, 0]).to(torch.float64).cpu().numpy()
    rows = np.repeat(batch.rows, np.diff(batch.offsets.astype(np.int64)))
    total = np.bincount(rows, weights=ln, minlength=case["files"])
    bp = np.rint(total[:, None] * cover[None, :] * noise).astype(np.int64)
    counts = np.where(empty, 0, np.maximum(1, bp // 500)).astype(np.int32)
    return counts, np.where(empty, 0, bp)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind in ("counts", "pairs"):
        cl, s["index"] = _index(case, seed)
        s["ctx"] = rg.Context(s["index"])
        s["files"] = _host_file(cl, seed, case["queries"], case["rows"])
        s["room"] = int(1.25 * _overlaps(case, case["queries"])[1]) + 1000
    elif kind == "batch":
        cl, s["index"] = _index(case, seed)
        s["ctx"] = rg.Context(s["index"])
        s["batch"], s["iv"] = _device_files(case, seed, cl)
        s["counts"] = torch.zeros((case["files"], s["index"].num_sources), dtype=torch.int32, device=DEV)
        s["bp"] = torch.zeros((case["files"], s["index"].num_sources), dtype=torch.int64, device=DEV)
    elif kind == "moments":
        s["store"] = api.Moments(1, [case["bins"]])
        s["iv"] = _moment_intervals(case, seed)
    else:
        cl, bins, cover, spread, _, _ = _pvalue_inputs(case, seed)
        s["store"] = api.Moments(case["sources"], bins)
        grids = [_moment_grid(int(b)).astype(np.float64) for b in bins]
        for d in range(case["sources"]):
            for c, g in enumerate(grids):
                s["store"].set(d, c, np.stack([cover[d] * g, cover[d] * spread[d] * g], 1))
        s["index"] = rg.Index.synth(rg.SynthSpec(3, cl, np.full(2, 1000, np.uint64)))
        s["ctx"] = rg.Context(s["index"])
        s["batch"], s["iv"] = _device_files(case, seed, cl)
        counts, bp = _observed(case, seed, s["batch"], s["iv"])
        s["counts"], s["bp"] = torch.from_numpy(counts).to(DEV), torch.from_numpy(bp).to(DEV)
        s["p"], s["llr"], s["lp"] = (torch.zeros(counts.shape, dtype=torch.float64, device=DEV) for _ in range(3))
        s["flags"] = torch.zeros(counts.shape, dtype=torch.uint8, device=DEV)
    return s


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "counts":
        counts, bp, _ = s["ctx"].query_counts(s["files"], case["rows"], with_overlap=case["overlap"])
        return (counts, bp) if case["overlap"] else (counts,)
    if kind == "pairs":
        pairs = s["ctx"].query_pairs(s["files"], case["rows"])
        n = len(pairs)
        pairs.resize((s["room"], 8), refcheck=False)  # as many rows for every seed; grown in place, zeros at the end
        return n, pairs
    if kind == "batch":
        s["ctx"].query_batch_device(s["batch"], s["counts"].data_ptr(), s["bp"].data_ptr(), graph=case["graph"], stats=False)
        return s["counts"], s["bp"]
    if kind == "moments":
        return s["store"].build(0, 0, s["iv"], case["bin"], report=True, precision=case["precision"])
    s["store"].batch_pvalues_device(s["ctx"], s["batch"], np.arange(CHROMS), s["counts"].data_ptr(), s["bp"].data_ptr(),
                                    s["p"].data_ptr(), s["llr"].data_ptr(), s["lp"].data_ptr(), s["flags"].data_ptr(),
                                    bin_size=PV_BIN, count_groups=False)
    return s["p"], s["llr"], s["lp"], s["flags"]


# ---- the work of a pass -----------------------------------------------------------------------------
def _overlaps(case, queries):
    """(expected database intervals that any query overlaps, expected overlapping pairs), from the length mix."""
    genome = float(rg.synth_chrom_lengths(1, CHROMS).sum())
    z = np.clip(np.exp(math.log(500.0) + np.sort(np.random.default_rng(0).normal(size=4096))), 20, 100_000)
    lens, w = z, np.full(z.shape, 1.0 / z.size)
    if case["db_files"] == 1000:
        b = np.exp(np.linspace(math.log(1e4), math.log(1e6), 512))
        lens, w = np.concatenate([z, b]), np.concatenate([0.95 * w, np.full(b.shape, 0.05 / b.size)])
    rate = queries * (lens + z.mean()) / genome
    return case["db_intervals"] * float((w * -np.expm1(-rate)).sum()), case["db_intervals"] * float((w * rate).sum())


def work(case):
    """Each interval read once (12 bytes), database intervals that no query overlaps not at all, each output written
    once; `flops`: two additions for each overlapping pair, or the arithmetic of the transforms and sums."""
    kind = case["kind"]
    if kind in ("counts", "pairs"):
        touched, hits = _overlaps(case, case["queries"])
        out = 32 * hits if kind == "pairs" else case["rows"] * case["db_files"] * (12 if case["overlap"] else 4)
        return {"bytes": 12.0 * (touched + case["queries"]) + out, "flops": 2.0 * hits}
    files = case.get("files", 0)
    queries = files * (case.get("largest", 1) - 100) / max(1e-9, math.log(max(2, case.get("largest", 1)) / 100.0))
    if kind == "batch":
        touched, hits = _overlaps(case, queries)
        return {"bytes": 12.0 * (touched + queries + files * case["db_files"]), "flops": 2.0 * hits}
    if kind == "moments":
        m = 2.0 ** math.ceil(math.log2(2 * case["bins"]))
        grid = len(_moment_grid(case["bins"]))
        return {"bytes": 12.0 * case["intervals"] + 24.0 * grid, "flops": 5.0 * m * math.log2(m) + 20.0 * case["bins"]}
    cells = files * case["sources"]
    groups = CHROMS * min(queries / files / CHROMS, 100.0)  # distinct lengths in bins of one file
    return {"bytes": 12.0 * queries + 37.0 * cells + 8.0 * case["sources"] * 2000.0, "flops": 8.0 * cells * groups}


# ---- the same in 64 bits ----------------------------------------------------------------------------
def _depth(iv, bins, size):
    """The coverage signal, which is defined in 32 bits in a fixed order: impulses bin by bin (starts, then ends, in
    file order), then prefix sums in chunks of eight with a running carry."""
    g = np.zeros(bins, np.float32)
    for sign, x in ((1, iv[:, 0]), (-1, iv[:, 1])):
        x = np.minimum(x.astype(np.int64), bins * size)
        b = x // size
        frac = (x % size).astype(np.float32) / np.float32(size)
        at = np.stack([b, np.where(frac > 0, b + 1, bins)], 1).ravel()
        val = np.stack([np.float32(1) - frac, frac], 1).ravel() * np.float32(sign)
        np.add.at(g, at[at < bins], val[at < bins])
    full = bins // 8
    body = np.add.accumulate(g[:8 * full].reshape(full, 8), axis=1, dtype=np.float32)
    carry = np.add.accumulate(body[:, 7], dtype=np.float32)
    body[1:] += carry[:-1, None]
    tail = np.add.accumulate(g[8 * full:], dtype=np.float32)
    return np.concatenate([body.ravel(), tail + carry[-1] if len(tail) else tail]).astype(np.float32)


def _exact_moments(case, seed):
    g = _depth(_moment_intervals(case, seed), case["bins"], case["bin"]).astype(np.longdouble)
    mean = g.sum() / case["bins"]
    u = np.concatenate([[0], np.cumsum(g - mean)]).astype(np.float64)
    u = torch.from_numpy(u).to(DEV if torch.cuda.is_available() else "cpu")
    means, varis = [], []
    for length in _moment_grid(case["bins"]).tolist():
        f = u[length:] - u[:-length]
        m = f.mean()
        means.append(length * float(mean) + float(m))
        varis.append(float((f - m).square().mean()))
    return np.array(means), np.array(varis)


def _tail(x):
    """ln(erfc(x) / 2) by the rational form 7.1.26 of Abramowitz and Stegun, which the path is defined with."""
    t = 1.0 / (1.0 + 0.3275911 * x)
    p = t * (0.254829592 + t * (-0.284496736 + t * (1.421413741 + t * (-1.453152027 + t * 1.061405429))))
    return np.log(0.5 * p) - x * x


def _exact_pvalues(case, seed):
    cl, bins, cover, spread, _, _ = _pvalue_inputs(case, seed)
    batch, iv = _device_files(case, seed, cl)
    counts, bp = _observed(case, seed, batch, iv)
    ln = (iv[:, 1] - iv[:, 0]).to(torch.float64).cpu().numpy() / PV_BIN
    cnt = np.diff(batch.offsets.astype(np.int64))
    rows, chrom = np.repeat(batch.rows, cnt), np.repeat(batch.shards, cnt).astype(np.int64)
    lint = np.maximum(1, np.ceil(ln)).astype(np.int64)
    ok = lint < bins[chrom].astype(np.int64)
    # the tables' entry of a length: the grid's, found as the store finds it
    far = lint > 100
    slot = np.where(far, 99 + np.floor(np.log(np.where(far, lint, 100) / 100.0) / np.log(1.01)).astype(np.int64), lint - 1)
    grid = [_moment_grid(int(b)) for b in bins]
    longest = max(grid, key=len)
    ok &= slot < np.array([len(g) for g in grid])[chrom]
    at = longest[np.where(ok, slot, 0)].astype(np.float64)
    # the tables hold 32-bit values: cover * L and cover * spread * L, rounded, for each source
    s = ln / lint
    key, inv = np.unique(np.where(ok, at, 0.0), return_inverse=True)
    n = len(key) * case["files"]
    where = (inv + rows.astype(np.int64) * len(key))[ok]
    s1, s2, s3 = (np.bincount(where, weights=v[ok], minlength=n).reshape(case["files"], -1) for v in (s, s * s, 1.0 / lint))
    mean = (cover[:, None] * key[None, :]).astype(np.float32).astype(np.float64)
    var = (cover[:, None] * spread[:, None] * key[None, :]).astype(np.float32).astype(np.float64)
    mu, v, raw = s1 @ mean.T, s2 @ var.T, s3 @ mean.T
    obs = bp / float(PV_BIN)
    some = counts > 0
    with np.errstate(all="ignore"):
        r, pp = mu * mu / (v - mu), mu / v
        po = r / (r + obs)
        nb = obs * np.log((1 - po) / (1 - pp)) + r * np.log(po / pp)
        oc = obs * raw / mu
        po_llr = oc * np.log(oc / raw) - (oc - raw)
        nb_ok = (mu > 0) & (pp > 0) & (pp < 1) & (po > 0) & (po < 1)
        po_ok = (raw > 0) & (oc > 0)
        llr = np.where(v > mu, np.where(nb_ok, nb, 0.0), np.where(po_ok, po_llr, 0.0))
        llr = np.where(some, llr, 0.0)
        lt = _tail(np.sqrt(np.maximum(llr, 0)))
        lp = np.where(llr > 0, np.where(obs >= mu, lt, np.log1p(-np.exp(lt))), 0.0)
        p = np.where(llr > 0, np.where(obs >= mu, np.exp(lt), 1.0 - np.exp(lt)), 1.0)
    return p, llr, lp, None


def exact(case, seed):
    """Counts, base pairs and pairs are whole numbers: nothing to say about them."""
    if case["kind"] == "moments":
        return _exact_moments(case, seed)
    if case["kind"] == "pvalues":
        return _exact_pvalues(case, seed)
    return None
