"""k_claim's wide shape (2,048 entries a step, where a call is costed and its queries average 4,096 and more)
in self-joins and R-S joins against the CPU oracle.  A record of more than 640 probe tokens makes the call a
costed one.  Pairs, overlaps and counters are whole numbers and must be equal."""
import numpy as np
import pytest

import new_fgssjoin_b200 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with F.Context(device=0) as c:
        yield c


def _sets(recs, n_terms):
    recs = sorted(recs, key=len, reverse=True)
    lens = np.array([len(r) for r in recs])
    pos = np.concatenate([[0], np.cumsum(lens[:-1])])
    return F.Sets(np.arange(1, len(recs) + 1), pos, lens, np.concatenate(recs).astype(np.uint32), n_terms)


def _long(rng, vocab):
    base = np.sort(rng.choice(vocab, 1400, replace=False))
    return [base, base[3:], base[:-2]]


def _wide(stats, queries):
    """k_cost_mj's average over the queries, by its window entries alone, is past the rule's 4,096."""
    assert stats["window_entries"] > 4096 * 1.1 * queries


@pytest.mark.parametrize("n", [4100, 6000])
def test_self_join_of_equal_records(ctx, n):
    """Windows of every multiple of the matches per source up to many steps."""
    rng = np.random.default_rng(n)
    s = _sets(_long(rng, 9000) + [np.arange(6)] * n, 9000)
    ref, st = O.join(s.pos, s.len, s.tokens, s.n_terms, 0.5)
    got = ctx.selfjoin(s, 0.5, method="batched")
    _wide(got.stats, n)
    assert np.array_equal(got.q, ref["q"]) and np.array_equal(got.s, ref["s"])
    assert np.array_equal(got.overlap, ref["overlap"])
    for k in ("candidates", "intersections", "results"):
        assert got.stats[k] == st[k], k


@pytest.mark.parametrize("vocab,t,nr,ns", [(60, 0.6, 5000, 7000), (300, 0.5, 14000, 16000)])
def test_rs_join(ctx, vocab, t, nr, ns):
    rng = np.random.default_rng(nr)
    pool = [np.sort(rng.choice(vocab, int(rng.integers(12, 30)), replace=False)) for _ in range(ns)]
    pick = [pool[int(i)][rng.random(len(pool[int(i)])) > 0.1] for i in rng.integers(0, ns, nr)]
    r = _sets([p for p in pick if len(p)] + _long(rng, 9000), 9000)
    s = _sets(pool + _long(rng, 9000), 9000)
    got = ctx.rsjoin(r, s, t, method="batched")
    _wide(got.stats, nr + ns)
    ref, st = O.rsjoin((r.pos, r.len, r.tokens), (s.pos, s.len, s.tokens), 9000, t)
    assert len(ref) > 0
    assert np.array_equal(got.q, ref["r"]) and np.array_equal(got.s, ref["s"])
    assert np.array_equal(got.overlap, ref["overlap"])
    for k in ("candidates", "intersections", "results"):
        assert got.stats[k] == st[k], k
