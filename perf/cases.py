"""Performance cases of the set-similarity join: what a program using this library has it do.

A case is one call (or one batched call) through the Python entry points, from the
latency-bound small join to the largest workload the benchmark defines.  The record
shapes are the repository's own workloads (new_fgssjoin_b200/datagen.py): Zipf-worded
titles, heavy-tailed records with near-duplicate clusters, and genome reads; they are
generated here with torch on the GPU so that fresh inputs are cheap to make.  A case has one
corpus; a seed renames its letters (for reads, its bases) and shuffles its records, so every
seed has other bytes, term ids and record orders, and the same number of similar pairs.

A program keeps one Context and hands it new inputs, so all cases of a process share one.
"""
import functools
import math

import numpy as np
import torch

import new_fgssjoin_b200 as F
from new_fgssjoin_b200.binding import _View

TITLE_TOK = dict(q=3, mode="qgram", pad=True, suffix=False, lower=True)
OCCUR_TOK = dict(q=3, mode="qgram", pad=False, suffix=True, lower=True)
READ_TOK = dict(q=16, mode="kmer", pad=False, suffix=False, lower=True)

# distinct 3-grams (k-mers), tokens with the occurrence suffix and text bytes per record
TOKENS = {"titles": 70, "heavy": 105, "reads": 135}
BYTES = {"titles": 75, "heavy": 147, "reads": 151}


# --------------------------------------------------------------------- cases
def listed():
    def join(name, data, n, t, method="batched", device=False, model=False, bounds="reference"):
        return dict(name=name, kind="join", data=data, n=n, t=t, method=method, device=device, model=model,
                    bounds=bounds)

    return [
        # interactive deduplication of a small list: the call's own latency
        join("titles1k_t80", "titles", 1000, 0.8, bounds="exact"),
        # the size and threshold of the reference's shipped title file, with the entry point's default method
        join("titles18k_t90_plain", "titles", 18000, 0.9, method="plain"),
        # a mid-sized title file joined at the default method
        join("titles100k_t70_plain", "titles", 100003, 0.7, method="plain"),
        # the benchmark's 100,000 titles at its lowest threshold, records already on the device
        join("titles100k_t50", "titles", 100000, 0.5, device=True),
        # the flagship: 1,000,000 heavy-tailed records on the device, with the trained cost model
        join("heavy1m_t70", "heavy", 1000000, 0.7, device=True, model=True),
        # a ragged count of long records from host arrays, exact rational bounds
        join("heavy150k_t85", "heavy", 149993, 0.85, bounds="exact"),
        # overlapping genome reads as canonical 16-mers, host arrays
        join("reads500k_t80", "reads", 500000, 0.8, bounds="exact"),
        # many independent joins of very different sizes in one call
        dict(name="batch48", kind="batch", joins=48, lo=1000, hi=50000),
        # two title files against each other
        dict(name="rs2x60k_t60", kind="rs", n=60000, t=0.6),
        # preprocessing: text to token sets, in the three forms the command line offers
        dict(name="tok_titles200k", kind="tok", data="titles", n=200000, form="distinct"),
        dict(name="tok_heavy60k_occ", kind="tok", data="heavy", n=60001, form="occurrence"),
        dict(name="tok_reads200k", kind="tok", data="reads", n=200000, form="kmer"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def join(data, n, t, method, device, model=False):
        # at 0.6 and 0.8 the reference's float32 bounds drop some pairs of exactly t, which ones by the term order
        return dict(kind="join", data=data, n=n, t=t, method=method, device=device, model=model,
                    bounds=rng.choice(["exact"] if t in (0.6, 0.8) else ["reference", "reference", "exact"]))

    kind = rng.choice(["titles", "titles", "heavy", "reads", "plain", "batch", "rs", "tok"])
    if kind == "titles":
        return join("titles", size(500, 200000), rng.choice([0.5, 0.6, 0.7, 0.8, 0.9, 0.95]), "batched",
                    rng.random() < 0.5)
    if kind == "heavy":
        return join("heavy", size(2000, 700000), rng.choice([0.7, 0.75, 0.8, 0.9]), "batched", rng.random() < 0.5,
                    rng.random() < 0.5)
    if kind == "reads":
        return join("reads", size(5000, 700000), rng.choice([0.7, 0.8, 0.9]), "batched", rng.random() < 0.5)
    if kind == "plain":
        return join("titles", size(500, 100000), rng.choice([0.6, 0.7, 0.8, 0.9]), "plain", False)
    if kind == "batch":
        return dict(kind="batch", joins=rng.randint(2, 48), lo=size(200, 2000), hi=size(4000, 50000))
    if kind == "rs":
        return dict(kind="rs", n=size(1000, 100000), t=rng.choice([0.6, 0.7, 0.8, 0.9]))
    data, form, hi = rng.choice([("titles", "distinct", 300000), ("titles", "occurrence", 300000),
                                 ("heavy", "distinct", 150000), ("heavy", "occurrence", 100000),
                                 ("reads", "kmer", 300000)])
    return dict(kind="tok", data=data, n=size(1000, hi), form=form)


def _batch_joins(case):
    """Sizes (log-uniform between lo and hi) and thresholds of a batch's joins: the same for every seed."""
    k = case["joins"]
    step = (math.log(case["hi"]) - math.log(case["lo"])) / max(1, k - 1)
    sizes = [int(round(case["lo"] * math.exp(step * ((i * 29) % k)))) for i in range(k)]
    return sizes, [(0.6, 0.7, 0.8, 0.9, 0.95)[i % 5] for i in range(k)]


def work(case):
    """Bytes of the records read once and of the pairs (or token sets) written once."""
    if case["kind"] == "tok":
        n, d = case["n"], case["data"]
        per = BYTES[d] if case["form"] == "occurrence" else TOKENS[d]
        return {"bytes": n * (BYTES[d] + 8 * per + 12), "flops": 0}
    if case["kind"] == "batch":
        n, d = sum(_batch_joins(case)[0]), "titles"
    elif case["kind"] == "rs":
        n, d = 2 * case["n"], "titles"
    else:
        n, d = case["n"], case["data"]
    return {"bytes": n * (12 + 4 * TOKENS[d] + 24 * 0.1), "flops": 0}


# -------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _titles_corpus(n, heavy):
    """Records of words drawn Zipf(1.1) from 50,000 words of 3-10 letters, one per line; some are copies of
    another record with 1-3 character substitutions (titles: 10 % of the records copy one other record;
    heavy: word counts lognormal(2.5, 1) in 2..600 and 5 % of the records in clusters of 2-20)."""
    g, dev = _gen(2 * n + heavy), "cuda"
    nv = 50000
    vlen = torch.randint(3, 11, (nv,), generator=g, device=dev)
    vchr = torch.randint(97, 123, (nv, 10), generator=g, device=dev, dtype=torch.uint8)
    cdf = torch.cumsum(torch.arange(1, nv + 1, device=dev, dtype=torch.float64) ** -1.1, 0)
    if heavy:
        z = torch.randn(n, generator=g, device=dev, dtype=torch.float64)
        wpr = torch.exp(2.5 + z).round().clamp(2, 600).long()
    else:
        wpr = torch.randint(5, 16, (n,), generator=g, device=dev)
    nw = int(wpr.sum())
    u = torch.rand(nw, generator=g, device=dev, dtype=torch.float64) * cdf[-1]
    wid = torch.searchsorted(cdf, u, right=True).clamp(max=nv - 1)
    # copies: record dup[i] becomes record base[i] with edits (bases are never copies)
    perm = torch.randperm(n, generator=g, device=dev)
    if heavy:
        m = n // 20
        sizes = torch.randint(2, 21, (m + 1,), generator=g, device=dev)
        start = torch.cumsum(sizes, 0) - sizes
        first = start[torch.searchsorted(start, torch.arange(m, device=dev), right=True) - 1]
        keep = torch.arange(m, device=dev) != first
        dup, base = perm[:m][keep], perm[first][keep]
    else:
        m = n // 10
        dup = perm[:m]
        base = perm[m:][torch.randint(0, n - m, (m,), generator=g, device=dev)]
    src = torch.arange(n, device=dev)
    src[dup] = base
    # words of every record, then the characters of every word, each word followed by one separator
    first_word = (torch.cumsum(wpr, 0) - wpr)[src]
    w = wid[_ragged(first_word, wpr[src])]
    wl = vlen[w] + 1
    wend = torch.cumsum(wl, 0)
    text = vchr.view(-1)[_ragged(w * 10, wl).clamp(max=10 * nv - 1)]
    text[wend - 1] = 32
    rend = wend[torch.cumsum(wpr[src], 0) - 1]  # end of every record, its separator included
    rbeg = torch.cat([rend.new_zeros(1), rend[:-1]])
    text[rend - 1] = 10
    edits = torch.randint(1, 4, (dup.numel(),), generator=g, device=dev)
    span = (rend - rbeg)[dup] - 1
    for k in range(3):
        at = rbeg[dup] + (torch.rand(dup.numel(), generator=g, device=dev, dtype=torch.float64) * span).long()
        ch = torch.randint(97, 123, (dup.numel(),), generator=g, device=dev, dtype=torch.uint8)
        text[at[edits > k]] = ch[edits > k]
    return text


def _reads_corpus(n):
    """150-base reads at random offsets of a random genome ten times as long as the reads, 0.5 % substitutions."""
    g, dev = _gen(n), "cuda"
    glen = 10 * n + 150
    genome = torch.randint(0, 4, (glen,), generator=g, device=dev, dtype=torch.uint8)
    start = torch.randint(0, glen - 149, (n,), generator=g, device=dev)
    r = genome[start[:, None] + torch.arange(150, device=dev)[None, :]]
    sub = torch.rand((n, 150), generator=g, device=dev) < 0.005
    r = torch.where(sub, (r + torch.randint(1, 4, (n, 150), generator=g, device=dev, dtype=torch.uint8)) % 4, r)
    out = torch.full((n, 151), 10, device=dev, dtype=torch.uint8)
    out[:, :150] = torch.tensor([65, 67, 71, 84], device=dev, dtype=torch.uint8)[r.long()]
    return out.view(-1)


def _ragged(start, count):
    """The concatenated ranges [start[i], start[i] + count[i])."""
    end = torch.cumsum(count, 0)
    return torch.repeat_interleave(start - (end - count), count, output_size=int(end[-1])) + \
        torch.arange(int(end[-1]), device=start.device)


@functools.lru_cache(maxsize=64)
def _corpus(data, n):
    """A case's records: their text and the first byte and byte count (newline included) of every line."""
    text = _reads_corpus(n) if data == "reads" else _titles_corpus(n, data == "heavy")
    end = torch.nonzero(text == 10).view(-1) + 1
    beg = torch.cat([end.new_zeros(1), end[:-1]])
    return text, beg, end - beg


def _text(data, n, seed, part=slice(None)):
    """Lines `part` of the corpus, shuffled, with its letters renamed (bases: a renaming that keeps the
    complements, so the canonical k-mers of two reads agree where they did)."""
    text, beg, cnt = _corpus(data, n)
    g = _gen(seed)
    lut = torch.arange(256, device="cuda", dtype=torch.uint8)
    if data == "reads":
        lut[torch.tensor([65, 67, 71, 84], device="cuda")] = torch.tensor(
            [list(x) for x in (b"ACGT", b"TCGA", b"AGCT", b"TGCA", b"CATG", b"CTAG", b"GATC", b"GTAC")],
            device="cuda", dtype=torch.uint8)[seed % 8]
    else:
        lut[97:123] = 97 + torch.randperm(26, generator=g, device="cuda").to(torch.uint8)
    beg, cnt = beg[part], cnt[part]
    order = torch.randperm(beg.numel(), generator=g, device="cuda")
    return lut[text[_ragged(beg[order], cnt[order])].long()].cpu().numpy().tobytes()


# ------------------------------------------------------- the program's handle
@functools.lru_cache(maxsize=None)
def _ctx():
    return F.Context(device=0)


@functools.lru_cache(maxsize=None)
def _trained(data, t):
    """Trains the context's cost model once, as a program does before it joins many inputs of one kind."""
    tok = READ_TOK if data == "reads" else TITLE_TOK
    sets = [_ctx().tokenize(_text(data, n, n), **tok) for n in (20000, 40000)]
    _ctx().model_train(sets, [t] * len(sets), epochs=200, lr=0.01, seed=1)


def _device_view(sets):
    """The records in device memory, as a caller that keeps its data there passes them."""
    cols = [torch.from_numpy(a.view(np.int32)).cuda() for a in (sets.id, sets.pos, sets.len, sets.tokens)]
    torch.cuda.synchronize()
    v = _View()
    v.id, v.pos, v.len, v.tokens = [c.data_ptr() for c in cols]
    v.n_sets, v.n_tokens, v.n_terms, v.on_device = sets.n_sets, sets.n_tokens, sets.n_terms, 1
    return v, cols


def prepare(case, seed):
    ctx = _ctx()
    st = {"case": case, "ctx": ctx}
    if case["kind"] == "tok":
        st["text"] = _text(case["data"], case["n"], seed)
    elif case["kind"] == "batch":
        sizes, st["ts"] = _batch_joins(case)
        st["sets"] = [ctx.tokenize(_text("titles", n, seed + i), **TITLE_TOK) for i, n in enumerate(sizes)]
    elif case["kind"] == "rs":
        st["r"], st["s"] = ctx.tokenize_dual(*_rs_texts(case, seed), **TITLE_TOK)
    else:
        tok = READ_TOK if case["data"] == "reads" else TITLE_TOK
        sets = ctx.tokenize(_text(case["data"], case["n"], seed), **tok)
        if case["model"]:
            _trained(case["data"], case["t"])
        if case["device"]:
            st["sets"], st["keep"] = _device_view(sets)
        else:
            st["sets"] = sets
    return st


def _rs_texts(case, seed):
    """One corpus of titles dealt alternately into the two files, so that copies meet across them."""
    n = 2 * case["n"]
    return _text("titles", n, seed, slice(0, None, 2)), _text("titles", n, seed, slice(1, None, 2))


# ----------------------------------------------------------------- one pass
def _pairs_out(p):
    return {"q": p.q, "s": p.s, "id_q": p.id_q, "id_s": p.id_s, "overlap": p.overlap, "sim": p.sim,
            "counts": [p.stats[k] for k in ("candidates", "intersections", "results", "index_entries")]}


def run(st):
    case, ctx = st["case"], st["ctx"]
    if case["kind"] == "tok":
        opts = {"distinct": TITLE_TOK, "occurrence": OCCUR_TOK, "kmer": READ_TOK}[case["form"]]
        s = ctx.tokenize(st["text"], **opts)
        return {"id": s.id, "pos": s.pos, "len": s.len, "tokens": s.tokens, "loc": s.loc, "n_terms": s.n_terms}
    if case["kind"] == "batch":
        res = ctx.selfjoin_batch(st["sets"], st["ts"], method="batched", bounds="exact")
        out = {k: np.concatenate([getattr(p, k) for p in res])  # one table of all pairs, as a program collects them
               for k in ("q", "s", "id_q", "id_s", "overlap", "sim")}
        out["counts"] = np.array([[p.stats[k] for k in ("candidates", "results")] for p in res], dtype=np.int64)
        return out
    if case["kind"] == "rs":
        return _pairs_out(ctx.rsjoin(st["r"], st["s"], case["t"], method="batched", bounds="exact"))
    return _pairs_out(ctx.selfjoin(st["sets"], case["t"], method=case["method"], bounds=case["bounds"],
                                   use_model=case["model"]))


# ---------------------------------------------------- the similarity in 64 bits
def _line_sets(text):
    """0/1 matrix (lines x distinct padded 3-grams, bfloat16) and the sizes of the lines' gram sets."""
    b = torch.frombuffer(bytearray(text), dtype=torch.uint8).cuda()
    end = torch.nonzero(b == 10).view(-1)
    beg = torch.cat([torch.zeros(1, device="cuda", dtype=torch.long), end[:-1] + 1])
    ln = end - beg
    n = ln.numel()
    g = ln + 2
    tot = int(g.sum())
    line = torch.repeat_interleave(torch.arange(n, device="cuda"), g, output_size=tot)
    i = torch.arange(tot, device="cuda") - (torch.cumsum(g, 0) - g)[line]
    key = torch.zeros(tot, device="cuda", dtype=torch.long)
    for k in range(3):
        at = i + k - 2
        inside = (at >= 0) & (at < ln[line])
        c = torch.where(inside, b[(beg[line] + at).clamp(0, b.numel() - 1)].long(), torch.ones_like(at))
        key = key * 256 + c
    uniq, ids = torch.unique(key, return_inverse=True)
    m = torch.zeros((n, uniq.numel()), device="cuda", dtype=torch.bfloat16)
    m[line, ids] = 1
    return m, m.sum(1, dtype=torch.float32).long()


def _similar(rows, rsize, cols, csize, t, upper):
    """overlap / union of every pair of a row and a column at or above t, ordered by (row, column)."""
    found = []
    step = 2048
    t32 = torch.tensor(t, dtype=torch.float32).item()
    for b in range(0, rows.shape[0], step):
        c0 = b if upper else 0
        o = torch.mm(rows[b:b + step], cols[c0:].T, out_dtype=torch.float32)
        u = rsize[b:b + step, None].float() + csize[None, c0:].float() - o
        hit = (o / u) >= t32
        if upper:
            hit &= torch.arange(c0, cols.shape[0], device="cuda")[None, :] > \
                torch.arange(b, b + o.shape[0], device="cuda")[:, None]
        r, c = torch.nonzero(hit, as_tuple=True)
        found.append(o[r, c].double() / u[r, c].double())
    return torch.cat(found)


def exact(case, seed):
    """The similarities in 64 bits from dense set products (small enough vocabularies and record counts only)."""
    if case["kind"] == "tok" or case.get("data") == "reads" or case.get("data") == "heavy" and case["n"] > 60000:
        return None

    def memory_order(m, size):
        # descending size, later lines first among equal sizes: the order of the records of a join
        o = torch.argsort(size * m.shape[0] + torch.arange(m.shape[0], device="cuda"), descending=True)
        return m[o], size[o]

    def selfjoin(text, t):
        m, size = memory_order(*_line_sets(text))
        return _similar(m, size, m, size, t, True)

    if case["kind"] == "rs":
        tr, ts = _rs_texts(case, seed)
        m, size = _line_sets(tr + ts)
        k = tr.count(b"\n")
        r, rs = memory_order(m[:k], size[:k])
        s, ss = memory_order(m[k:], size[k:])
        sim = _similar(r, rs, s, ss, case["t"], False)
    elif case["kind"] == "batch":
        sim = torch.cat([selfjoin(_text("titles", n, seed + i), t)
                         for i, (n, t) in enumerate(zip(*_batch_joins(case)))])
    else:
        sim = selfjoin(_text(case["data"], case["n"], seed), case["t"])
    return {"sim": sim.cpu().numpy()}
