"""The strategy that the autotuner reports, asked for by name, runs what it had timed: the same
kernels as the automatic choice, and the same pairs."""
import numpy as np
import pytest

import new_fgssjoin_b200 as F
from new_fgssjoin_b200 import datagen

pytestmark = pytest.mark.gpu


def _same(a, b):
    for k in ("q", "s", "overlap", "sim"):
        assert np.array_equal(getattr(a, k), getattr(b, k)), k
    for k in ("candidates", "intersections", "results"):
        assert a.stats[k] == b.stats[k], k


def test_reported_strategy_runs_the_tuned_variant(tmp_path):
    path = str(tmp_path / "tune.json")
    with F.Context(device=0, tune_cache_path=path) as c:
        s = c.tokenize(datagen.titles(20000, seed=3), **datagen.TITLE_TOK)
        named = c.selfjoin(s, 0.5, method="batched", filter="warp")  # nothing tuned yet
        best = c.autotune(s, 0.5, reps=2)
        auto = c.selfjoin(s, 0.5, method="batched")
        got = c.selfjoin(s, 0.5, method="batched", filter=best["filter"])
        assert got.stats["launches"] == auto.stats["launches"]
        _same(got, auto)
        _same(named, auto)
        for other in {"warp", "cta", "global"} - {best["filter"]}:  # the others as they are named
            p = c.selfjoin(s, 0.5, method="batched", filter=other)
            _same(p, auto)
            assert (p.stats["heavy_queries"] > 0) == (other == "global")
        # a batch of both ways of asking
        res = c.selfjoin_batch([s, s], [0.5, 0.5], method="batched", filter=best["filter"])
        _same(res[0], auto)
        _same(res[1], auto)
    with F.Context(device=0, tune_cache_path=path) as c:  # from the cache file
        got = c.selfjoin(s, 0.5, method="batched", filter=best["filter"])
        assert got.stats["launches"] == c.selfjoin(s, 0.5, method="batched").stats["launches"]
        _same(got, auto)


def test_device_arrays_replay_it(tmp_path):
    """Recorded, captured and replayed with the strategy asked for by name."""
    import torch
    from new_fgssjoin_b200.binding import _View
    with F.Context(device=0) as c:
        s = c.tokenize(datagen.titles(20000, seed=4), **datagen.TITLE_TOK)
        best = c.autotune(s, 0.5, reps=2)
        cols = [torch.from_numpy(a.view(np.int32)).cuda() for a in (s.id, s.pos, s.len, s.tokens)]
        torch.cuda.synchronize()
        v = _View()
        v.id, v.pos, v.len, v.tokens = [x.data_ptr() for x in cols]
        v.n_sets, v.n_tokens, v.n_terms, v.on_device = s.n_sets, s.n_tokens, s.n_terms, 1
        want = c.selfjoin(s, 0.5, method="batched")
        for _ in range(3):
            _same(c.selfjoin(v, 0.5, method="batched", filter=best["filter"]), want)
