"""The claim kernels (k_claim, k_tiny) against the CPU oracle at the edges of their
routes: window entries around k_tiny's 128 and a step's 2048, id windows inside and
across the block table's 4096-id blocks, many matches per source, vocabularies around
the membership bitmap's 32,768 terms, probe prefixes around 640 tokens, unsorted
records and both sides of an R-S join.  Pairs, overlaps and counters are whole numbers
and must be equal."""
import numpy as np
import pytest

import new_fgssjoin_b200 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with F.Context(device=0) as c:
        yield c


def _sets(recs, n_terms, sort=True):
    if sort:
        recs = sorted(recs, key=len, reverse=True)
    lens = np.array([len(r) for r in recs])
    pos = np.concatenate([[0], np.cumsum(lens[:-1])])
    return F.Sets(np.arange(1, len(recs) + 1), pos, lens, np.concatenate(recs).astype(np.uint32), n_terms)


def _check(got, s, t):
    ref, st = O.join(s.pos, s.len, s.tokens, s.n_terms, t)
    assert np.array_equal(got.q, ref["q"]) and np.array_equal(got.s, ref["s"])
    assert np.array_equal(got.overlap, ref["overlap"])
    for k in ("candidates", "intersections", "results"):
        assert got.stats[k] == st[k], k
    return ref


@pytest.mark.parametrize("n", [2, 33, 44, 65, 130, 700, 1100])
def test_identical_records(ctx, n):
    """n equal records of 6 tokens: the window of record q holds a multiple of n - q - 1 entries, each
    source matched several times, so every entry count up to several steps occurs."""
    s = _sets([np.arange(6)] * n, 6)
    ref = _check(ctx.selfjoin(s, 0.5, method="batched"), s, 0.5)
    assert len(ref["q"]) == n * (n - 1) // 2


@pytest.mark.parametrize("n", [4095, 4097, 8193])
@pytest.mark.parametrize("vocab,t", [(40, 0.6), (400, 0.5), (33000, 0.5)])
def test_blocks_of_ids(ctx, n, vocab, t):
    """Windows inside one block of ids and across several, from dense (a few dozen terms) to sparse."""
    rng = np.random.default_rng(n + vocab)
    base = [np.sort(rng.choice(vocab, int(rng.integers(3, 24)), replace=False)) for _ in range(n // 3)]
    recs = []
    for i in range(n):
        b = base[int(rng.integers(0, len(base)))]
        recs.append(np.unique(np.concatenate([b[rng.random(len(b)) > 0.15], rng.choice(vocab, 2, replace=False)])))
    s = _sets(recs, vocab)
    _check(ctx.selfjoin(s, t, method="batched"), s, t)


@pytest.mark.parametrize("size", [1100, 1279, 1300])
def test_long_probe_prefixes(ctx, size):
    """Records whose probe prefix (about half their size at t = 0.5) lies around 640 tokens."""
    rng = np.random.default_rng(size)
    base = np.sort(rng.choice(40000, size, replace=False))
    recs = [base[rng.random(size) > 0.05] for _ in range(150)]
    recs += [np.sort(rng.choice(40000, 30, replace=False)) for _ in range(200)]
    s = _sets(recs, 40000)
    _check(ctx.selfjoin(s, 0.5, method="batched"), s, 0.5)


def test_unsorted_records_across_blocks(ctx):
    rng = np.random.default_rng(5)
    recs = [np.sort(rng.choice(300, int(rng.integers(4, 20)), replace=False)) for _ in range(5000)]
    for i in range(0, 5000, 3):
        recs[i] = recs[(i * 7) % 5000]
    s = _sets(recs, 300, sort=False)
    _check(ctx.selfjoin(s, 0.6, method="batched"), s, 0.6)


@pytest.mark.parametrize("nr,ns", [(3000, 4000), (60, 90)])
def test_rs_join(ctx, nr, ns):
    rng = np.random.default_rng(nr)
    pool = [np.sort(rng.choice(500, int(rng.integers(4, 30)), replace=False)) for _ in range(ns)]
    pick = [pool[int(i)][rng.random(len(pool[int(i)])) > 0.1] for i in rng.integers(0, ns, nr)]
    r, s = _sets([p for p in pick if len(p)], 500), _sets(pool, 500)
    got = ctx.rsjoin(r, s, 0.6, method="batched")
    ref = ctx.rsjoin(r, s, 0.6, method="plain")
    assert len(ref) > 0
    for k in ("q", "s", "overlap", "sim"):
        assert np.array_equal(getattr(got, k), getattr(ref, k)), k
    assert got.stats["candidates"] == ref.stats["candidates"]


def test_replay_on_other_contents(ctx):
    """A captured call replayed after its device arrays changed from short windows to long ones."""
    import torch
    from new_fgssjoin_b200.binding import _View
    rng = np.random.default_rng(3)
    n, L = 5000, 12
    a = np.sort(np.stack([rng.choice(4000, L, replace=False) for _ in range(n)]), axis=1)
    b = np.sort(np.stack([rng.choice(60, L, replace=False) for _ in range(n)]), axis=1)
    cols = [torch.from_numpy(x.astype(np.int32)).cuda() for x in
            (np.arange(1, n + 1), np.arange(n) * L, np.full(n, L), a.reshape(-1))]
    torch.cuda.synchronize()
    v = _View()
    v.id, v.pos, v.len, v.tokens = [c.data_ptr() for c in cols]
    v.n_sets, v.n_tokens, v.n_terms, v.on_device = n, n * L, 4000, 1
    for x in (a, a, b, b, a):
        cols[3].copy_(torch.from_numpy(x.reshape(-1).astype(np.int32)))
        torch.cuda.synchronize()
        s = F.Sets(np.arange(1, n + 1), np.arange(n) * L, np.full(n, L), x.reshape(-1).astype(np.uint32), 4000)
        _check(ctx.selfjoin(v, 0.7, method="batched"), s, 0.7)
