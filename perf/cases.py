"""The work that users of this framework have it do, as cases that can be timed.

A case is a plain dict: its kind, its sizes and its options.  `prepare` makes
what a program holds before the call (a resident index, a batch handle, the
queries in host memory), `run` is one pass through the public entry points,
`exact` is the same answer from plain torch in 64 bits and `work` the bytes
and additions that a pass cannot do without.

Kinds:
  range   byte-valued tables (half-normal, 30 % zeros), one value per object
          and dim; queries of exact or range items, counts or weighted scores
  lsh     hash-bucket signatures: many short lists, exact items
  text    compressed posting lists of Zipf terms, decoded while counting
  bag     bag-of-words rows (a row lists any number of terms)
  build   the inverted index built from a value matrix
  decode  encoded posting segments decoded on the device
"""
import ctypes
import math

import numpy as np
import torch

import genie_gb300 as genie

ZERO_FRAC, SIGMA = 0.30, 40.0
TEXT_CODEC = 13            # delta, then BP32 blocks with a varint tail
RADII = (0, 1, 2, 4)


def listed():
    return [
        # one interactive lookup in a small table: latency and launches only
        dict(name="lookup_1k", kind="range", n=1000, d=128, q=1, m_lo=128, m_hi=128, radius=0, weights="none",
             k_lo=10, k_hi=10, entry="search"),
        # the quick-start size: a hundred exact queries against a thousand objects
        dict(name="small_100q", kind="range", n=1000, d=128, q=100, m_lo=128, m_hi=128, radius=0, weights="none",
             k_lo=10, k_hi=10, entry="search"),
        # one uneven range query against a large table: an online request served alone
        dict(name="one_range_2m", kind="range", n=2_000_003, d=128, q=1, m_lo=90, m_hi=90, radius=2, weights="none",
             k_lo=100, k_hi=100, entry="search"),
        # an ordinary table and a request's worth of range queries, counts only
        dict(name="range_counts_260k", kind="range", n=260_000, d=128, q=256, m_lo=8, m_hi=128, radius=-1,
             weights="none", k_lo=10, k_hi=100, entry="search"),
        # the same with every query weighted: scores as well as counts
        dict(name="range_weighted_500k", kind="range", n=499_999, d=128, q=512, m_lo=8, m_hi=128, radius=-1,
             weights="all", k_lo=10, k_hi=100, entry="batch"),
        # the batched uneven workload: half the queries weighted, k 10 or 100, a large table
        dict(name="uneven_mixed_4m", kind="range", n=4_000_000, d=128, q=2048, m_lo=8, m_hi=128, radius=-1,
             weights="half", k_lo=10, k_hi=100, entry="batch"),
        # the LSH-style batch at its full size
        dict(name="lsh_batch_1m", kind="lsh", n=1_000_000, d=240, q=1024, k=100, buckets=8192, entry="batch"),
        # a few signatures looked up at once (plain call)
        dict(name="lsh_few_300k", kind="lsh", n=300_001, d=240, q=24, k=50, buckets=8192, entry="search"),
        # short texts over compressed lists, batched
        dict(name="text_1m", kind="text", n=1_000_000, d=32, q=1024, k=32, terms=65536, segment=128),
        # bag-of-words rows, as the tweets-like tables
        dict(name="bag_400k", kind="bag", n=400_000, q=200, m=10, k=20, terms=65536),
        # the index builder on byte values (long lists) and on hash buckets (short ones)
        dict(name="build_u8_1m", kind="build", n=1_000_000, d=128, values="u8"),
        # encoded segments decoded on the device
        dict(name="decode_64k", kind="decode", segments=65536, length=1024, codec=TEXT_CODEC),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["range", "range", "range", "range", "lsh", "lsh", "text", "bag", "build", "build", "decode"])
    if kind == "range":
        n = _log_int(rng, 1000, 4_000_000)
        q = _log_int(rng, 1, min(2048, max(1, int(4e9 / n))))
        m_hi = rng.randint(8, 128)
        exact = rng.random() < 0.2
        return dict(kind=kind, n=n, d=128, q=q, m_lo=rng.randint(4, 8), m_hi=m_hi,
                    radius=0 if exact else -1, weights=rng.choice(["none", "none", "half", "all"]), k_lo=10,
                    k_hi=rng.choice([10, 50, 100, 100, 500]), entry=rng.choice(["search", "batch"]))
    if kind == "lsh":
        n = _log_int(rng, 20_000, 1_000_000)
        return dict(kind=kind, n=n, d=rng.randint(32, 240), q=_log_int(rng, 1, 1024), k=rng.choice([10, 50, 100]),
                    buckets=rng.choice([1024, 4096, 8192]), entry=rng.choice(["search", "batch"]))
    if kind == "text":
        return dict(kind=kind, n=_log_int(rng, 50_000, 1_000_000), d=rng.randint(8, 32), q=_log_int(rng, 1, 1024),
                    k=rng.choice([10, 32, 100]), terms=rng.choice([4096, 65536]), segment=rng.choice([128, 128, 1024]))
    if kind == "bag":
        return dict(kind=kind, n=_log_int(rng, 2000, 400_000), q=_log_int(rng, 1, 400), m=rng.randint(3, 24),
                    k=rng.choice([5, 20, 50]), terms=rng.choice([4096, 65536]))
    if kind == "build":
        values = rng.choice(["u8", "lsh"])
        cells = _log_int(rng, 1_000_000, 120_000_000)
        d = rng.randint(8, 128)
        return dict(kind=kind, n=max(1000, cells // d), d=d, values=values)
    return dict(kind=kind, segments=_log_int(rng, 100, 65536), length=rng.choice([128, 1024, rng.randint(1, 1024)]),
                codec=rng.choice([TEXT_CODEC, 11, 10, 12, 4, 3]))


# ---------------------------------------------------------------- inputs

def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(1_000_003 * int(seed) + salt)
    return g


def _u8_values(n, d, g):
    """n x d half-normal byte values with 30 % zeros, as int32 on the GPU."""
    v = torch.randn((n, d), device="cuda", generator=g).mul_(SIGMA).abs_().round_().clamp_(max=255)
    v.masked_fill_(torch.rand((n, d), device="cuda", generator=g) < ZERO_FRAC, 0)
    return v.to(torch.int32)


def _zipf_p(terms, s=1.1):
    p = np.arange(1, terms + 1, dtype=np.float64) ** (-s)
    return p / p.sum()


def _zipf(shape, terms, g):
    cdf = torch.from_numpy(np.cumsum(_zipf_p(terms))).to("cuda", torch.float64)
    u = torch.rand(shape, device="cuda", generator=g, dtype=torch.float64)
    return torch.searchsorted(cdf, u).clamp_(max=terms - 1).to(torch.int32)


def _range_inputs(case, seed):
    """(values on the GPU, query arrays): items on distinct dims around the
    values of stored objects, half-width `radius` (-1: 0, 1, 2 or 4 per query; 0: exact items)."""
    n, d, q = case["n"], case["d"], case["q"]
    values = _u8_values(n, d, _gen(seed, 1))
    rng = np.random.default_rng([int(seed), 2])
    m = rng.integers(case["m_lo"], case["m_hi"] + 1, q) if case["m_hi"] > case["m_lo"] else np.full(q, case["m_hi"])
    m = np.minimum(m, d)
    off = np.zeros(q + 1, np.int64)
    off[1:] = np.cumsum(m)
    order = np.argsort(rng.random((q, d)), axis=1).astype(np.int32)
    take = np.arange(d)[None, :] < m[:, None]
    if (m == d).all():
        order = np.tile(np.arange(d, dtype=np.int32), (q, 1))
    dim = np.ascontiguousarray(order[take])
    src = torch.from_numpy(np.repeat(rng.integers(0, n, q), m)).cuda()
    centre = values[src, torch.from_numpy(dim.astype(np.int64)).cuda()].cpu().numpy()
    if case["radius"] == 0:      # exact items on perturbed values
        low = np.clip(centre + np.rint(rng.normal(0, 8, len(centre))), 0, 255).astype(np.int32)
        up = low
    else:
        r = np.repeat(rng.choice(np.array(RADII if case["radius"] < 0 else [case["radius"]], np.int32), q), m)
        low, up = centre - r, centre + r
    # one k for half of the queries and the other for the rest, in any order
    k = rng.permutation(np.array([case["k_lo"], case["k_hi"]], np.uint32)[np.arange(q) % 2])
    weight = weighted = None
    if case["weights"] != "none":
        weight = rng.uniform(0.5, 2.0, int(off[-1])).astype(np.float32)
        weighted = np.ones(q, np.uint8) if case["weights"] == "all" else (np.arange(q) % 2).astype(np.uint8)
    return values, dict(item_off=off, dim=dim, low=low, up=up, k=k, weight=weight, weighted=weighted)


def _lsh_inputs(case, seed):
    """Uniform buckets; half the queries are stored objects with 60 % of their
    items redrawn, half are uniform."""
    n, d, q = case["n"], case["d"], case["q"]
    values = torch.randint(0, case["buckets"], (n, d), device="cuda", generator=_gen(seed, 1), dtype=torch.int32)
    rng = np.random.default_rng([int(seed), 2])
    qv = rng.integers(0, case["buckets"], size=(q, d), dtype=np.int32)
    half = (q + 1) // 2
    src = values[torch.from_numpy(rng.integers(0, n, half)).cuda()].cpu().numpy()
    keep = rng.random((half, d)) >= 0.60
    qv[:half] = np.where(keep, src, qv[:half])
    low = np.ascontiguousarray(qv.ravel())
    return values, dict(item_off=np.arange(q + 1, dtype=np.int64) * d, dim=np.tile(np.arange(d, dtype=np.int32), q),
                        low=low, up=low, k=case["k"], weight=None, weighted=None)


def _text_inputs(case, seed):
    n, d, q = case["n"], case["d"], case["q"]
    values = _zipf((n, d), case["terms"], _gen(seed, 1))
    low = _zipf((q, d), case["terms"], _gen(seed, 2)).cpu().numpy().ravel()
    return values, dict(item_off=np.arange(q + 1, dtype=np.int64) * d, dim=np.tile(np.arange(d, dtype=np.int32), q),
                        low=low, up=low, k=case["k"], weight=None, weighted=None)


def _bag_inputs(case, seed):
    """Rows of 4 to 20 Zipf terms; a query holds m terms of one row and of the
    vocabulary, each once or more."""
    n, q, m = case["n"], case["q"], case["m"]
    rng = np.random.default_rng([int(seed), 3])
    length = rng.integers(4, 21, n)
    off = np.zeros(n + 1, np.int64)
    off[1:] = np.cumsum(length)
    values = _zipf((int(off[-1]),), case["terms"], _gen(seed, 1)).cpu().numpy()
    terms = _zipf((q, m), case["terms"], _gen(seed, 2)).cpu().numpy()
    row = rng.integers(0, n, q)
    at = off[row][:, None] + rng.integers(0, 1 << 30, (q, m)) % length[row][:, None]
    terms = np.where(rng.random((q, m)) < 0.6, values[at], terms)
    low = np.ascontiguousarray(terms.ravel().astype(np.int32))
    return (values, off), dict(item_off=np.arange(q + 1, dtype=np.int64) * m, dim=np.zeros(q * m, np.int32), low=low,
                               up=low, k=case["k"], weight=None, weighted=None)


def _build_inputs(case, seed):
    """A value matrix whose first and last rows hold the least and the greatest
    value (a black and a saturated image), so that every dim has all its lists."""
    g = _gen(seed, 1)
    if case["values"] == "u8":
        v = _u8_values(case["n"], case["d"], g)
    else:
        v = torch.randint(0, 8192, (case["n"], case["d"]), device="cuda", generator=g, dtype=torch.int32)
    v[0], v[-1] = 0, 255 if case["values"] == "u8" else 8191
    return v


def _decode_inputs(case, seed):
    """Sorted ids with geometric gaps, encoded segment by segment; a pool of
    distinct segments repeated to the size wanted.  The last one is short."""
    rng = np.random.default_rng([int(seed), 4])
    pool, length = min(512, case["segments"]), case["length"]
    lib = genie.lib()
    words, lens, ids = [], [], []
    buf = np.zeros(int(lib.genie_codec_encode_bound(1024)) + 64, np.uint32)
    for i in range(pool):
        n = length if i < pool - 1 or pool == 1 else max(1, length // 2)
        gap = rng.geometric(float(rng.choice([0.3, 0.05, 0.01, 0.001])), n)
        v = np.minimum(np.cumsum(gap) + int(rng.integers(0, 1 << 20)), (1 << 28) - 1).astype(np.uint32)
        w = lib.genie_codec_encode(case["codec"], v.ctypes.data, n, buf.ctypes.data, len(buf))
        if w <= 0:
            raise RuntimeError("encode failed")
        words.append(buf[:w].copy())
        lens.append(n)
        ids.append(v)
    reps = np.arange(case["segments"]) % pool
    word_len = np.array([len(w) for w in words], np.int64)[reps]
    seg_len = np.array(lens, np.int64)[reps]
    full, rest = divmod(case["segments"], pool)
    flat = np.concatenate([np.tile(np.concatenate(words), full)] + words[:rest])
    ids = np.concatenate([np.tile(np.concatenate(ids), full)] + ids[:rest])
    word_off = np.zeros(case["segments"] + 1, np.int64)
    out_off = np.zeros(case["segments"] + 1, np.int64)
    np.cumsum(word_len, out=word_off[1:])
    np.cumsum(seg_len, out=out_off[1:])
    return flat, word_off, out_off, seg_len, ids


_INPUTS = dict(range=_range_inputs, lsh=_lsh_inputs, text=_text_inputs, bag=_bag_inputs)


# ---------------------------------------------------------------- the passes

def prepare(case, seed):
    kind = case["kind"]
    if kind == "build":
        return dict(kind=kind, values=np.ascontiguousarray(_build_inputs(case, seed).cpu().numpy()))
    if kind == "decode":
        words, word_off, out_off, _, ids = _decode_inputs(case, seed)
        dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
        return dict(kind=kind, codec=case["codec"], n=case["segments"], words=dev(words.view(np.int32)),
                    word_off=dev(word_off), out_off=dev(out_off[:-1].copy()),
                    out=torch.zeros(len(ids), dtype=torch.int32, device="cuda"),
                    lens=torch.zeros(case["segments"], dtype=torch.int32, device="cuda"))
    rows, b = _INPUTS[kind](case, seed)
    queries = genie.QueryBatch(b["item_off"], b["dim"], b["low"], b["up"], b["k"], b["weight"], b["weighted"])
    if kind == "bag":
        table = genie.Table.from_bag_arrays(*rows)
    elif kind == "text":
        table = genie.Table.compressed(rows.cpu().numpy(), TEXT_CODEC, case["segment"])
    else:
        table = genie.Table.from_values(rows.cpu().numpy())
    del rows
    torch.cuda.empty_cache()
    batch = None
    if kind == "text" or case.get("entry") == "batch":
        batch = genie.Batch(table, queries.n_queries, len(queries.dim), int(queries.k_array.max()))
    return dict(kind=kind, table=table, batch=batch, queries=queries, scores=b["weight"] is not None)


def run(state):
    kind = state["kind"]
    if kind == "build":
        table = genie.Table.from_values(state["values"])
        layout, ids = table.layout(), table.ids()
        table.close()
        return dict(ids=ids.view(np.int32), **layout)
    if kind == "decode":
        rc = genie.lib().genie_codec_decode_device(
            state["codec"], state["words"].data_ptr(), state["word_off"].data_ptr(), state["n"],
            state["out_off"].data_ptr(), state["out"].data_ptr(), state["lens"].data_ptr(),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise RuntimeError(genie.lib().genie_last_error().decode())
        return [state["out"], state["lens"]]
    if state["batch"] is not None:
        return list(state["batch"].run(state["queries"], scores=state["scores"]))
    return list(genie.search(state["table"], state["queries"], scores=state["scores"]))


# ---------------------------------------------------------------- 64-bit answers

def _top(prim, k):
    """The k best objects by (prim desc, id asc) of one query: ids, prims; (0, 0) past the matches."""
    k_eff = min(k, prim.numel())
    if prim.dtype == torch.float64:
        val, at = torch.sort(prim, descending=True, stable=True)
        val, at = val[:k_eff], at[:k_eff]
    else:
        key = (prim.to(torch.int64) << 32) | (0xFFFFFFFF - torch.arange(prim.numel(), device=prim.device))
        key = torch.topk(key, k_eff).values
        val, at = key >> 32, 0xFFFFFFFF - (key & 0xFFFFFFFF)
    at = torch.where(val > 0, at, torch.zeros_like(at))
    pad = k - k_eff
    if pad:
        at, val = torch.cat([at, at.new_zeros(pad)]), torch.cat([val, val.new_zeros(pad)])
    return at, val


def exact(case, seed):
    kind = case["kind"]
    if kind == "decode":
        _, _, _, seg_len, ids = _decode_inputs(case, seed)
        return [torch.from_numpy(ids.astype(np.int64)), torch.from_numpy(seg_len)]
    if kind == "build":
        v = _build_inputs(case, seed).to(torch.int64)
        mn, mx = v.min(0).values, v.max(0).values
        base = torch.zeros(case["d"] + 1, dtype=torch.int64, device="cuda")
        base[1:] = torch.cumsum(mx - mn + 1, 0)
        count = torch.zeros(int(base[-1]) + 1, dtype=torch.int64, device="cuda")
        ids = torch.empty((case["d"], case["n"]), dtype=torch.int64, device="cuda")
        for j in range(case["d"]):
            ids[j] = torch.sort(v[:, j], stable=True).indices
            c = torch.bincount(v[:, j] - mn[j])
            count[int(base[j]) + 1:int(base[j]) + 1 + c.numel()] = c
        return dict(ids=ids.reshape(-1), key_offsets=torch.cumsum(count, 0), key_base=base, dim_min=mn, dim_max=mx)
    rows, b = _INPUTS[kind](case, seed)
    if kind == "bag":
        values, off = rows
        n = case["n"]
        obj = torch.from_numpy(np.repeat(np.arange(n), np.diff(off))).cuda()
        term = torch.from_numpy(values.astype(np.int64)).cuda()
    else:
        n = case["n"]
        cols = rows.t().contiguous().to(torch.int16 if kind == "lsh" else torch.uint8 if kind == "range" else torch.int32)
        del rows
        if n * len(b["dim"]) > 1.5e11 and b["weight"] is not None:
            return None
    ks = np.broadcast_to(np.asarray(b["k"], np.int64), (case["q"],))
    ids, prims = [], []
    for q in range(case["q"]):
        i0, i1 = int(b["item_off"][q]), int(b["item_off"][q + 1])
        weighted = b["weighted"] is not None and b["weighted"][q]
        acc = torch.zeros(n, dtype=torch.float64 if weighted else torch.int16, device="cuda")
        for i in range(i0, i1):
            lo, up = int(b["low"][i]), int(b["up"][i])
            if kind == "bag":
                acc += torch.bincount(obj[term == lo], minlength=n).to(torch.int16)
                continue
            c = cols[int(b["dim"][i])]
            lo, up = max(lo, 0), min(up, int(torch.iinfo(c.dtype).max))
            hit = (c == lo) if lo == up else ((c >= lo) & (c <= up))
            if weighted:
                acc.add_(hit, alpha=float(b["weight"][i]))
            else:
                acc += hit
        at, val = _top(acc, int(ks[q]))
        ids.append(at)
        prims.append(val.to(torch.float64))
    ids, prims = torch.cat(ids), torch.cat(prims)
    if b["weight"] is None:
        return [ids, prims.to(torch.int64)]
    # objects whose weighted sums agree to the last bits may rank either way, and a count is a cut score
    return [None, None, prims]


# ---------------------------------------------------------------- what a pass cannot do without

def _u8_p():
    z = np.arange(0, 256, dtype=np.float64)
    cdf = np.array([math.erf(x / (SIGMA * math.sqrt(2))) for x in np.append(z + 0.5, 0.0)])
    p = np.diff(np.concatenate([[0.0], cdf[:256]]))
    p[255] += 1 - cdf[255]
    p *= 1 - ZERO_FRAC
    p[0] += ZERO_FRAC
    return p


def work(case):
    """Bytes: the posting lists that the queries touch, each read once (no more
    than the index), the queries and the results; additions: one per posting id
    of every query.  An index build reads the values and writes the ids; a
    decode reads the words and writes the ids."""
    kind = case["kind"]
    if kind == "build":
        cells = case["n"] * case["d"]
        return dict(bytes=8.0 * cells, flops=0.0)
    if kind == "decode":
        cells = case["segments"] * case["length"]
        return dict(bytes=cells * (4.0 + 1.2), flops=float(cells))
    n, q = case["n"], case["q"]
    if kind == "range":
        p = _u8_p()
        m = 0.5 * (case["m_lo"] + case["m_hi"])
        c = np.concatenate([[0.0], np.cumsum(p)])
        v = np.arange(256)
        mean = lambda r: float(np.sum(p * (c[np.minimum(v + r, 255) + 1] - c[np.maximum(v - r, 0)])))  # noqa: E731
        hit = mean(case["radius"]) if case["radius"] >= 0 else sum(mean(r) for r in RADII) / len(RADII)
        per_query, index, per_id, k = m * n * hit, 4.0 * n * case["d"], 4.0, 0.5 * (case["k_lo"] + case["k_hi"])
    elif kind == "lsh":
        m, k, per_id = case["d"], case["k"], 4.0
        per_query, index = m * n / case["buckets"], 4.0 * n * case["d"]
    elif kind == "text":
        p = _zipf_p(case["terms"])
        m, k, per_id = case["d"], case["k"], 1.2
        per_query, index = m * n * float(np.sum(p * p)), 1.2 * n * case["d"]
    else:
        p = _zipf_p(case["terms"])
        m, k, per_id = case["m"], case["k"], 4.0
        per_query, index = m * n * 12 * float(np.sum(p * p)), 4.0 * n * 12
    results = q * k * (12.0 if case.get("weights", "none") != "none" else 8.0)
    return dict(bytes=min(index, q * per_query * per_id) + q * m * 12.0 + results, flops=float(q * per_query))
