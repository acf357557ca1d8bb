"""A wait between the tiles of a scan that runs out: the call fails with FGSS_ERR_TIMEOUT, nothing
is written past the output, and the context's next calls are right."""
import numpy as np
import pytest
import torch

import new_fgssjoin_b200 as F
from new_fgssjoin_b200 import datagen
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TIMEOUT = 7


@pytest.mark.parametrize("n", [4096, 4097, 8192, 4096 * 33 + 5, 4096 * 700 + 1])
def test_a_scan_without_polls(n):
    a = np.random.default_rng(n).integers(0, 1 << 20, n).astype(np.uint32)
    want = (np.cumsum(a.astype(np.uint64)) - a).astype(np.uint32)
    d = torch.from_numpy(a.view(np.int32)).cuda()
    out = torch.full((n + 64,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    with F.Context(device=0) as c:
        for _ in range(2):
            if n <= 4096:  # one tile: no wait
                c.dev_exclusive_scan_u32_polls(d.data_ptr(), out.data_ptr(), n, 0)
            else:
                with pytest.raises(F.FgssError) as e:
                    c.dev_exclusive_scan_u32_polls(d.data_ptr(), out.data_ptr(), n, 0)
                assert e.value.status == TIMEOUT
            got = out.cpu().numpy().view(np.uint32)
            assert np.array_equal(got[:4096], want[:4096]) and (got[n:] == 0xFFFFFFFF).all()
            c.dev_exclusive_scan_u32(d.data_ptr(), out.data_ptr(), n)
            assert np.array_equal(out.cpu().numpy().view(np.uint32)[:n], want)
        # kernels that look at the word run again
        s = c.tokenize(datagen.titles(3000, seed=7), **datagen.TITLE_TOK)
        ref, _ = O.join(s.pos, s.len, s.tokens, s.n_terms, 0.8)
        for method in ("batched", "plain"):
            p = c.selfjoin(s, 0.8, method=method)
            assert np.array_equal(p.q, ref["q"]) and np.array_equal(p.s, ref["s"])
