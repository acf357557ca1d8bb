"""Calls the library refuses, from a caller whose output struct holds whatever was there."""
import ctypes

import pytest

import new_fgssjoin_b200 as F
from new_fgssjoin_b200 import binding as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q,mode,suffix", [(0, 0, 0), (1025, 0, 0), (33, 1, 0), (7, 0, 1)])
def test_refused_tokenizer_options_leave_an_empty_struct(q, mode, suffix):
    """Nothing of an uninitialized fgss_sets is freed."""
    lib = F.load_library()
    with F.Context(device=0) as c:
        s = B._Sets()
        ctypes.memset(ctypes.byref(s), 0x5A, ctypes.sizeof(s))
        o = B._TokOpts(q, mode, 0, 1, suffix, 1)
        assert lib.fgss_tokenize(c._ctx, b"abcdefgh\n", 9, ctypes.byref(o), ctypes.byref(s)) != 0
        assert bytes(s) == bytes(ctypes.sizeof(s))
        assert c.tokenize(b"abcdefgh\n", q=3).n_sets == 1
