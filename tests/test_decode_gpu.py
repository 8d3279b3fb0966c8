"""Decoding on the device against the token-by-token loop: sizes either side of the tile, ids that the vocabulary does not have, entries
of no and of many bytes, a vocabulary that changes between calls, and the inputs that still go through the loop."""
import numpy as np
import pytest

from gpu_bpe_b200 import TrieTokenizer

pytestmark = pytest.mark.gpu

VOCAB = [bytes([i]) for i in range(256)] + [b"the ", b"x" * 300, "\u4f60\u597d".encode(), b"ab"]


def _loop(vocab, tokens) -> bytes:
    return b"".join(bytes(vocab[int(t)]) if int(t) < len(vocab) else b"\xef\xbf\xbd" for t in tokens)


@pytest.mark.parametrize("n", [0, 1, 3, 255, 1023, 1024, 1025, 4097, 300_001])
@pytest.mark.parametrize("top", [256, 260, 300, 2**32])
def test_sizes_and_unknown_ids(engine, n, top):
    tok = TrieTokenizer.fromVocab(engine, list(VOCAB))
    tokens = np.random.default_rng(n + top % 999).integers(0, top, n, dtype=np.uint32)
    assert tok.decode(tokens) == _loop(VOCAB, tokens)
    tok.destroy()


def test_more_bytes_than_expected(engine):
    tok = TrieTokenizer.fromVocab(engine, list(VOCAB))
    tokens = np.full(5000, 257, np.uint32)
    assert tok.decode(tokens) == b"x" * 1_500_000 and tok.decode(tokens[:7]) == b"x" * 2100
    tok.destroy()


def test_the_vocabulary_as_it_is_at_the_call(engine):
    vocab = list(VOCAB)
    tok = TrieTokenizer.fromVocab(engine, vocab)
    tokens = np.array([256, 97, 260, 259, 98], np.uint32)
    assert tok.decode(tokens) == _loop(vocab, tokens)
    vocab[259] = b"changed"
    vocab.append(b"new")
    assert tok.decode(tokens) == _loop(vocab, tokens) == b"the anewchangedb"
    vocab[256] = bytearray(b"THE")
    assert tok.decode(tokens) == _loop(vocab, tokens)
    vocab[256][0] = 0x74
    assert tok.decode(tokens) == b"tHEanewchangedb"
    vocab[97] = b""
    vocab[256] = b""
    assert tok.decode(tokens) == b"newchangedb"
    tok.destroy()
    assert tok.decode(tokens) == b"newchangedb"


def test_other_inputs(engine):
    tok = TrieTokenizer.fromVocab(engine, list(VOCAB))
    t = [256, 97, 999, 258]
    want = _loop(VOCAB, t)
    for x in (t, tuple(t), np.array(t), np.array(t, np.int16), np.array([t, t], np.uint32)[0], np.array(t * 2, np.uint32)[::2].repeat(1), iter(t)):
        x = list(x) if not isinstance(x, np.ndarray) and not isinstance(x, list) else x
        assert tok.decode(x) == _loop(VOCAB, x)
    assert tok.decode(t) == want and tok.decode(np.array([-1])) == VOCAB[-1]
    tok.destroy()
