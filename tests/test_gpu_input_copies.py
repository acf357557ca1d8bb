"""Token sets to the device in one copy (columns of one page-locked block) or four (any other
arrays): slices of a block's columns, plain arrays and mixtures of both give the oracle's pairs."""
import numpy as np
import pytest

import new_fgssjoin_b200 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["block", "plain", "mixed", "tail"])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 900])
def test_forms_of_host_arrays(form, n):
    rng = np.random.default_rng(n)
    words = [bytes(rng.choice(np.frombuffer(b"abcde", np.uint8), 12)) for _ in range(max(2, n // 3))]
    text = b"\n".join(words[int(i)] for i in rng.integers(0, len(words), n)) + b"\n"
    with F.Context(device=0) as ctx:
        a = ctx.tokenize(text, q=3, pad=False, suffix=False)
        cols = [a.id, a.pos, a.len, a.tokens]
        if form == "plain":
            cols = [c.copy() for c in cols]
        elif form == "mixed":
            cols[2] = cols[2].copy()
        elif form == "tail":  # the records from the second on: slices inside the block
            cols[:3] = [c[1:] for c in cols[:3]]
        if form == "tail" and n == 1:
            return
        s = F.Sets(cols[0], cols[1], cols[2], cols[3], a.n_terms)
        for method in ("batched", "plain"):
            got = ctx.selfjoin(s, 0.7, method=method)
            ref, st = O.join(s.pos, s.len, s.tokens, s.n_terms, 0.7)
            assert np.array_equal(got.q, ref["q"]) and np.array_equal(got.s, ref["s"])
            assert np.array_equal(got.overlap, ref["overlap"])
            assert got.stats["candidates"] == st["candidates"]
            assert np.array_equal(got.id_q, s.id[got.q]) and np.array_equal(got.id_s, s.id[got.s])
