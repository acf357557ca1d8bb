"""Joins without per-query costs and work items, and the plain method's stages, against
the CPU oracle: both query classes of the claim kernels and the keyed table behind them,
few and many verification records (a warp takes 1 to 32 of them; above 65,536 the number
of results is waited for), the wanted candidates, and a captured call replayed on records
whose probe prefixes no longer fit it.  Whole numbers, which must be equal."""
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


def _corpus(n, vocab, seed, lo=3, hi=24):
    rng = np.random.default_rng(seed)
    base = [np.sort(rng.choice(vocab, int(rng.integers(lo, hi)), replace=False)) for _ in range(max(1, n // 3))]
    recs = []
    for _ in range(n):
        b = base[int(rng.integers(0, len(base)))]
        recs.append(np.unique(np.concatenate([b[rng.random(len(b)) > 0.15], rng.choice(vocab, 2, replace=False)])))
    return recs


@pytest.mark.parametrize("method", ["plain", "batched"])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 32, 33, 255, 256, 257, 1185, 2369, 9473])
def test_sizes(ctx, method, n):
    """Record counts around the tiles (8 to 256 records) and the item sizes of the kernels."""
    s = _sets(_corpus(n, 300, n), 300)
    _check(ctx.selfjoin(s, 0.6, method=method), s, 0.6)


@pytest.mark.parametrize("n", [130, 363, 700, 1100])
def test_plain_identical_records(ctx, n):
    """n (n - 1) / 2 results: 8,385 to 604,450, on both sides of 65,536, every record merged."""
    s = _sets([np.arange(6)] * n, 6)
    ref = _check(ctx.selfjoin(s, 0.5, method="plain"), s, 0.5)
    assert len(ref["q"]) == n * (n - 1) // 2


@pytest.mark.parametrize("size", [1100, 1279, 1280, 1281, 1300])
def test_plain_long_probe_prefixes(ctx, size):
    """Probe prefixes (about half of 1100 to 1300 tokens at t = 0.5) around the claim kernel's 640."""
    rng = np.random.default_rng(size)
    base = np.sort(rng.choice(40000, size, replace=False))
    recs = [base] + [base[rng.random(size) > 0.05] for _ in range(150)]
    recs += [np.sort(rng.choice(40000, 30, replace=False)) for _ in range(200)]
    s = _sets(recs, 40000)
    for method in ("plain", "batched"):
        _check(ctx.selfjoin(s, 0.5, method=method), s, 0.5)


def test_plain_unsorted(ctx):
    recs = _corpus(5000, 300, 5)
    s = _sets(recs, 300, sort=False)
    _check(ctx.selfjoin(s, 0.6, method="plain"), s, 0.6)


def test_replay_after_records_grew(ctx):
    """A call captured on short records, replayed when the same arrays hold records beyond 640 probe tokens."""
    import torch
    from new_fgssjoin_b200.binding import _View
    rng = np.random.default_rng(7)
    n, total, vocab = 600, 60000, 5000
    short = [np.sort(rng.choice(vocab, 100, replace=False)) for _ in range(n)]
    longs = [np.sort(rng.choice(vocab, 1400, replace=False))]
    longs += [np.sort(np.unique(np.concatenate([longs[0][:1390], rng.choice(vocab, 10)]))) for _ in range(19)]
    left = total - sum(len(r) for r in longs)
    per = left // (n - 20)
    longs += [np.sort(rng.choice(vocab, per, replace=False)) for _ in range(n - 20)]
    longs[-1] = np.sort(rng.choice(vocab, per + total - sum(len(r) for r in longs), replace=False))
    longs.sort(key=len, reverse=True)
    a, b = _sets(short, vocab), _sets(longs, vocab)
    cols = [torch.from_numpy(np.asarray(x).astype(np.int32)).cuda() for x in (a.id, a.pos, a.len, a.tokens)]
    torch.cuda.synchronize()
    v = _View()
    v.id, v.pos, v.len, v.tokens = [c.data_ptr() for c in cols]
    v.n_sets, v.n_tokens, v.n_terms, v.on_device = n, total, vocab, 1
    for s in (a, a, b, b, a):
        assert len(s.tokens) == total
        for c, x in zip(cols, (s.id, s.pos, s.len, s.tokens)):
            c.copy_(torch.from_numpy(np.asarray(x).astype(np.int32)))
        torch.cuda.synchronize()
        _check(ctx.selfjoin(v, 0.5, method="batched"), s, 0.5)


@pytest.mark.parametrize("n", [1500, 5000])
def test_claim_shapes(ctx, n):
    """One record with a probe prefix beyond 640, so the costs are read back: below and above an
    average of 4,096 window entries a query the claim kernel's two shapes run (about 1,800 and 6,000)."""
    rng = np.random.default_rng(n)
    recs = [np.sort(rng.choice(5000, 2600, replace=False))]
    recs += [np.sort(rng.choice(40, 24, replace=False)) for _ in range(n)]
    s = _sets(recs, 5000)
    got = ctx.selfjoin(s, 0.7, method="batched")
    assert (got.stats["window_entries"] / n >= 4096) == (n == 5000)
    _check(got, s, 0.7)
