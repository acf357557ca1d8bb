"""Contexts on several threads at once: calls that share the library's kernels, each from its
own context, give what they give alone (whole numbers)."""
import threading

import numpy as np
import pytest

import new_fgssjoin_b200 as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("suffix", [False, True])
def test_tokenize_lines_of_several_sizes_beside_each_other(suffix):
    """Lines of 3,000 and of 8,000 grams take tables of different sizes (64 and 128 KB of shared memory)."""
    rng = np.random.default_rng(1)
    texts = [bytes(rng.choice(np.frombuffer(b"abcdefghijklmnopqrstuvwxyz ", np.uint8), n)) for n in (3000, 8000)]
    opts = dict(q=3, pad=False, suffix=suffix)
    with F.Context(device=0) as c:
        want = [c.tokenize(t, **opts) for t in texts]
    failed = []

    def work(k):
        try:
            with F.Context(device=0) as c:
                for _ in range(300):
                    got = c.tokenize(texts[k], **opts)
                    for a in ("id", "pos", "len", "tokens", "loc"):
                        assert np.array_equal(getattr(got, a), getattr(want[k], a)), a
        except Exception as e:  # noqa: BLE001
            failed.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(i % 2,)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert failed == []
