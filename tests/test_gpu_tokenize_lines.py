"""The line-by-line tokenizer at the edges of its classes (lines and records of 256, 1024
and 8192 grams, the last with the global-sort pipeline beyond it), of its gram codes and of
the text's own layout, against the oracle (whole numbers)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(ctx, text, **opts):
    s = ctx.tokenize(text, **opts)
    ids, lens, tok, loc, nt = O.tokenize(text, **opts)
    mid, mpos, mlen, mtok = O.file_to_memory(ids, lens, tok)
    _, _, _, mloc = O.file_to_memory(ids, lens, loc)
    assert s.n_terms == nt
    assert np.array_equal(s.id, mid) and np.array_equal(s.len, mlen) and np.array_equal(s.pos, mpos)
    assert np.array_equal(s.tokens, mtok)
    assert np.array_equal(s.loc, mloc) if len(mtok) else s.loc is None  # (no column without tokens)


def _line(rng, n, alphabet):
    return bytes(rng.choice(np.frombuffer(alphabet, np.uint8), n).astype(np.uint8))


@pytest.mark.parametrize("grams", [1, 31, 32, 33, 64, 255, 256, 257, 1023, 1024, 1025, 2500, 8191, 8192, 8193])
@pytest.mark.parametrize("suffix", [False, True])
def test_line_lengths(ctx, grams, suffix):
    rng = np.random.default_rng(grams)
    lines = [_line(rng, grams + 2, a) for a in (b"ab", b"abcdefghijklmnopqrstuvwxyz ", bytes(range(32, 127)))]
    lines += [_line(rng, int(n), b"abc de") for n in rng.integers(1, 60, 40)]
    _check(ctx, b"\n".join(lines) + b"\n", q=3, pad=False, suffix=suffix, lower=True)


@pytest.mark.parametrize("q,pad,suffix,pad_char", [(1, True, True, 1), (2, True, False, 97), (3, True, False, 200),
                                                   (4, False, True, 1), (6, True, True, 32), (7, True, False, 1),
                                                   (8, True, False, 1)])
@pytest.mark.parametrize("alphabet", [b"a", b"aAbB", bytes(set(range(256)) - {10})], ids=["a", "aAbB", "all"])
def test_gram_codes(ctx, q, pad, suffix, pad_char, alphabet):
    rng = np.random.default_rng(q)
    text = b"\n".join(_line(rng, int(n), alphabet) for n in rng.integers(0, 90, 300))
    for lower in (True, False):
        _check(ctx, text, q=q, pad=pad, suffix=suffix, pad_char=pad_char, lower=lower)


@pytest.mark.parametrize("k", [1, 5, 16, 17, 31, 32])
def test_kmers(ctx, k):
    rng = np.random.default_rng(k)
    lines = [_line(rng, int(n), b"ACGTacgt") for n in rng.integers(1, 400, 200)]
    lines += [b"T" * 80, b"A" * 80, b"ACGT" * 30, b"N" * 40, b"ACGTNNACGTACGTAGCTAGCTAGCTAGCTAGCTAGCATCGATC" * 3]
    lines += [_line(rng, 700, b"ACGTN") for _ in range(5)] + [_line(rng, 3000, b"ACGT") for _ in range(3)]
    _check(ctx, b"\n".join(lines), q=k, mode="kmer", pad=False, suffix=False)


@pytest.mark.parametrize("text", [b"abc", b"\nabc", b"abc\n", b"\n\n\nabcd\n\n\nabce\n\n", b"\n" * 5000 + b"hello world",
                                  b"x" * 4095 + b"\n" + b"y" * 4096 + b"\n" + b"z" * 4097, b"ab\n" * 9000,
                                  b"abcdefgh\r\n" * 700], ids=range(8))
def test_text_layout(ctx, text):
    _check(ctx, text, q=3, pad=True, suffix=False, lower=True)
    _check(ctx, text, q=3, pad=False, suffix=True, lower=True)


@pytest.mark.parametrize("sizes", [[256] * 4096, [256] * 4095 + [255], [8192] * 128,
                                   [8000] * 3 + [1000] * 40 + [500] * 200 + [60] * 15500],
                         ids=["2^20", "2^20-1", "long", "mixed"])
def test_result_in_parts(ctx, sizes):
    """Results of 2^20 tokens and more go to the host in parts of 1, 2, 4 and 8 fifteenths of the records."""
    rng = np.random.default_rng(len(sizes))
    lines = [_line(rng, n + 2, b"abcdefghijklmnopqrstuvwxyz ") for n in rng.permutation(sizes)]
    _check(ctx, b"\n".join(lines), q=3, pad=False, suffix=True, lower=True)
