"""A tokenizer mode other than the two named ones is k-mers, as it always was: the same limit on k, the
same token sets."""
import ctypes

import numpy as np
import pytest

import fake_util
import new_fgssjoin_b200 as F
from new_fgssjoin_b200 import binding as B


def test_modes_of_the_options(tmp_path):
    out = fake_util.run(tmp_path, r"""
#include <stdio.h>
#include <string.h>
#include "tokenize.h"
void fgss_tok_opts_default(fgss_tok_opts* o) { *o = fgss_tok_opts{3, FGSS_TOK_QGRAM, 0, 1, 1, 1}; }
int main() {
    for (int mode : {0, 1, 2, -1, 256}) {
        const fgss_tok_opts o{16, mode, 1, 'x', 0, 0};
        const fgss::TokParams p = fgss::tok_params(&o);
        printf("%d %d %d %d %d %d\n", p.q, p.mode, p.pad, p.pad_char, p.suffix, p.lower);
    }
    const fgss::TokParams p = fgss::tok_params(nullptr);
    printf("%d %d %d %d %d %d\n", p.q, p.mode, p.pad, p.pad_char, p.suffix, p.lower);
}
""").splitlines()
    assert out == ["16 0 1 120 0 0"] + ["16 1 1 120 0 0"] * 4 + ["3 0 0 1 1 1"]


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [2, -1])
def test_other_modes_are_kmers(mode):
    lib = F.load_library()
    rng = np.random.default_rng(mode & 7)
    reads = [bytes(rng.choice(np.frombuffer(b"ACGTacgtN", np.uint8), n)) for n in (1, 20, 33, 90, 400, 1500)] * 3
    text = b"\n".join(reads)
    with F.Context(device=0) as c:
        def tokenize(q, m):
            s = B._Sets()
            o = B._TokOpts(q, m, 1, 65, 1, 0)
            return lib.fgss_tokenize(c._ctx, text, len(text), ctypes.byref(o), ctypes.byref(s)), s
        for q in (3, 9, 16, 32):
            got = []
            for m in (mode, 1):
                st, s = tokenize(q, m)
                assert st == 0
                got.append(F.Sets._from_c(s))
            for k in ("id", "pos", "len", "tokens", "loc"):
                assert np.array_equal(getattr(got[0], k), getattr(got[1], k)), (q, k)
        assert tokenize(33, mode)[0] == tokenize(33, 1)[0] != 0
