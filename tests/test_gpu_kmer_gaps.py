"""k-mers of lines with other bytes than A/C/G/T between them, whose windows are skipped: terms of one
document frequency are numbered by first occurrence whatever the length of the text's longest line
(8,192 windows are the line tokenizer's limit; beyond, the text takes the global sorts)."""
import numpy as np
import pytest

import new_fgssjoin_b200 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("longest", [200, 8192, 9000, 30000])
@pytest.mark.parametrize("q", [1, 3, 11, 17, 32])
def test_first_occurrence_order(longest, q):
    rng = np.random.default_rng(longest + q)
    base = bytes(rng.choice(np.frombuffer(b"ACGTNacgt-", np.uint8), longest + q - 1,
                            p=[.2, .2, .2, .2, .01, .04, .04, .04, .04, .03]))
    lens = rng.integers(1, 300, 40)
    lines = [base[int(a):int(a) + int(n)] for a, n in zip(rng.integers(0, max(1, len(base) - 300), 40), lens)]
    text = b"\n".join(lines[:20] + [base, b"N" * 50] + lines[20:])
    ids, ln, tok, _, nt = O.tokenize(text, q=q, mode="kmer")
    mid, mpos, mlen, mtok = O.file_to_memory(ids, ln, tok)
    with F.Context(device=0) as c:
        got = c.tokenize(text, q=q, mode="kmer")
    assert got.n_terms == nt
    for a, b in ((got.id, mid), (got.pos, mpos), (got.len, mlen), (got.tokens, mtok)):
        assert np.array_equal(a, b)
