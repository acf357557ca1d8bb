"""The plain method's verification against the CPU oracle where a warp's candidate records lie in groups
(a record above 256 tokens in the join) and where they do not, from one record a warp to 32, with runs of
near-duplicates among them.  Pairs, overlaps and counters are whole numbers and must be equal."""
import numpy as np
import pytest

import new_fgssjoin_b200 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with F.Context(device=0) as c:
        yield c


@pytest.mark.parametrize("longest", [40, 256, 257, 3000])
@pytest.mark.parametrize("n,vocab", [(3, 60), (120, 60), (1500, 60), (4000, 50)])
def test_groups_of_records(ctx, n, vocab, longest):
    rng = np.random.default_rng(n + longest)
    short = [np.sort(rng.choice(vocab, int(rng.integers(8, 25)), replace=False)) for _ in range(n)]
    base = np.sort(rng.choice(8000, longest, replace=False))
    dups = [np.delete(base, rng.choice(longest, longest // 20, replace=False)) for _ in range(40)]
    recs = sorted(short + [base] + dups, key=len, reverse=True)
    lens = np.array([len(r) for r in recs])
    s = F.Sets(np.arange(1, len(recs) + 1), np.concatenate([[0], np.cumsum(lens[:-1])]), lens,
               np.concatenate(recs).astype(np.uint32), 8000)
    ref, st = O.join(s.pos, s.len, s.tokens, s.n_terms, 0.6)
    got = ctx.selfjoin(s, 0.6, method="plain")
    assert np.array_equal(got.q, ref["q"]) and np.array_equal(got.s, ref["s"])
    assert np.array_equal(got.overlap, ref["overlap"])
    for k in ("candidates", "intersections", "results"):
        assert got.stats[k] == st[k], k
    if n == 4000:
        assert st["candidates"] > 32 * 64 * 148  # 32 records a warp
