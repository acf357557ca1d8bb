"""The plain method where its queries divide between k_probe and the claim kernels: probe prefixes around
384 tokens in joins with and without one above 640, queries around k_probe's 2048 tokens, and those of the
global accumulator, whose launches run beside each other.  Against the CPU oracle, in whole numbers, call
after call on one context."""
import numpy as np
import pytest

import new_fgssjoin_b200 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with F.Context(device=0) as c:
        yield c


def _sets(sizes, vocab, seed):
    rng = np.random.default_rng(seed)
    recs = []
    for z in sizes:
        base = np.sort(rng.choice(vocab, z, replace=False))
        recs += [base] + [np.delete(base, rng.choice(z, max(1, z // 12), replace=False)) for _ in range(6)]
    recs += [np.sort(rng.choice(vocab, 30, replace=False)) for _ in range(150)]
    recs.sort(key=len, reverse=True)
    lens = np.array([len(r) for r in recs])
    return F.Sets(np.arange(1, len(recs) + 1), np.concatenate([[0], np.cumsum(lens[:-1])]), lens,
                  np.concatenate(recs).astype(np.uint32), vocab)


@pytest.mark.parametrize("sizes,t", [
    ((700, 767, 768, 770, 900), 0.5),            # prefixes around 384, none above 640
    ((700, 767, 768, 770, 1279, 1281), 0.5),     # and one above it
    ((1500, 2040, 2049, 2100, 3300), 0.8),       # queries around 2048 tokens
    ((400, 900, 1400, 2300, 5000), 0.6),         # some on the global accumulator
])
@pytest.mark.parametrize("vocab", [9000, 60000])
def test_classes(ctx, sizes, t, vocab):
    s = _sets(sizes, vocab, len(sizes) + vocab)
    ref, st = O.join(s.pos, s.len, s.tokens, s.n_terms, t)
    assert st["results"] > 0
    for _ in range(3):
        got = ctx.selfjoin(s, t, method="plain")
        assert np.array_equal(got.q, ref["q"]) and np.array_equal(got.s, ref["s"])
        assert np.array_equal(got.overlap, ref["overlap"])
        for k in ("candidates", "intersections", "results"):
            assert got.stats[k] == st[k], k


def test_both_sides(ctx):
    r, s = _sets((700, 1300), 9000, 1), _sets((700, 1300, 2300), 9000, 2)
    a, b = (ctx.rsjoin(r, s, 0.5, method=m) for m in ("plain", "batched"))
    for k in ("q", "s", "overlap", "sim"):
        assert np.array_equal(getattr(a, k), getattr(b, k)), k
    assert a.stats["candidates"] == b.stats["candidates"]
