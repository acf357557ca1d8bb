"""Query ranges of a join (first records of pairs) that begin and end anywhere: one query, inside a tile of
records, across several, up to the last record.  The pairs are those of the whole join with their first
record in the range, and ranges that cover the join add up to its counters."""
import numpy as np
import pytest

import new_fgssjoin_b200 as F

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with F.Context(device=0) as c:
        yield c


def _sets(n, seed, longest):
    """n records over a small vocabulary, some of them equal; `longest` tokens in the first three."""
    rng = np.random.default_rng(seed)
    pool = [np.sort(rng.choice(300, int(rng.integers(4, 20)), replace=False)) for _ in range(max(1, n // 2))]
    recs = [pool[int(i)] for i in rng.integers(0, len(pool), n)]
    if longest:
        base = np.sort(rng.choice(30000, longest, replace=False))
        recs[:3] = [base, base[1:], base[:-1]]
    recs.sort(key=len, reverse=True)
    lens = np.array([len(r) for r in recs])
    pos = np.concatenate([[0], np.cumsum(lens[:-1])])
    return F.Sets(np.arange(1, n + 1), pos, lens, np.concatenate(recs).astype(np.uint32), 30000)


@pytest.mark.parametrize("longest", [0, 1500])
@pytest.mark.parametrize("method", ["batched", "plain"])
@pytest.mark.parametrize("n", [3, 300, 20000])
def test_ranges(ctx, n, method, longest):
    s = _sets(n, n + longest, longest)
    full = ctx.selfjoin(s, 0.6, method=method)
    cuts = sorted({x for x in (0, 1, 2, n // 3, n // 3 + 1, 255, 256, 257, 8191, 8192, 12345, n - 1, n) if x <= n})
    total = {"candidates": 0, "intersections": 0, "results": 0, "window_entries": 0}
    for a, b in zip(cuts[:-1], cuts[1:]):
        got = ctx.selfjoin(s, 0.6, method=method, query_range=(a, b))
        keep = (full.q >= a) & (full.q < b)
        for k in ("q", "s", "overlap", "sim"):
            assert np.array_equal(getattr(got, k), getattr(full, k)[keep]), (a, b, k)
        for k in total:
            total[k] += got.stats[k]
    assert total == {k: full.stats[k] for k in total}
