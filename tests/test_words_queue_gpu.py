"""Merges with more occurrences in the dictionary than the queues in shared memory hold (65,536 list entries make a second round): the
occurrences that wait outside them, for pairs of equal symbols in runs of 2 to 300 at every alignment, for pairs of different ones, for
pairs of merged symbols, in both compaction modes, against the pass-by-pass oracle."""
import numpy as np
import pytest

from tests.test_words_gpu import _check as check_fixed
from tests.test_words_literal_gpu import _check as check_literal

pytestmark = pytest.mark.gpu

ROUND = 65536


def _distinct_words(n_words, body, seed, pad=17):
    """Words `up to pad - 1 x + body + number`, all of them distinct, in random order: data, mask, and the words."""
    rng = np.random.default_rng(seed)
    words = []
    for i in range(n_words):
        number, digits = i, []
        while True:                                          # in letters c..z, least significant first
            digits.append(99 + number % 24)
            number //= 24
            if number == 0:
                break
        words.append(bytes([120] * (i % pad)) + body(rng) + bytes(digits))
    order = rng.permutation(n_words)
    data = np.frombuffer(b"".join(words[i] for i in order), np.uint8)
    mask = np.zeros(data.size, np.uint8)
    mask[np.cumsum([0] + [len(words[i]) for i in order[:-1]])] = 1
    return data, mask, words


def _occurrences(words, pair):
    return sum(w[k:k + 2] == pair for w in set(words) for k in range(len(w) - 1))


@pytest.mark.parametrize("longest", [2, 3, 7, 300])
def test_runs_of_equal_symbols_fixed(engine, longest):
    runs = lambda rng: b"a" * int(rng.integers(2, longest + 1)) if longest > 2 else b"aa"
    data, mask, words = _distinct_words({2: 80_000, 3: 60_000, 7: 30_000, 300: 3_000}[longest], runs, longest)
    assert _occurrences(words, b"aa") > ROUND
    check_fixed(engine, data, mask, 12)


@pytest.mark.parametrize("body,pair", [(b"ab", b"ab"), (b"abab", b"ab"), (b"abaabba", b"ab"), (b"abababab", b"ba")])
def test_different_and_merged_symbols_fixed(engine, body, pair):
    """`abababab`: the second merge is of two equal merged symbols."""
    data, mask, words = _distinct_words(70_000, lambda rng: body, len(body))
    assert _occurrences(words, pair) > ROUND
    check_fixed(engine, data, mask, 12)


@pytest.mark.parametrize("equal", [True, False])
def test_literal(engine, equal):
    """Words of random letters around the pair, so that its count stays within the tail of a "literal" run."""
    def body(rng):
        w = rng.integers(97, 123, size=60).astype(np.uint8).tobytes()
        return w[:30] + (b"A" * int(rng.integers(2, 6)) if equal else b"ABAB") + w[30:]
    data, mask, words = _distinct_words(60_000, body, 5 + equal, pad=1)
    assert _occurrences(words, b"AA" if equal else b"AB") > ROUND * 32 // 28
    check_literal(engine, data, mask, [1, 2, 6])
