"""The segment kernel of the merge-replay encoder at the sizes where it can go wrong, against the CPU oracle: segment lengths
either side of a thread's and a warp's share and of the longest that is taken, texts either side of the tile edges, rules over
ids that nothing makes, and the number of rules that were applied."""
import numpy as np
import pytest

from gpu_bpe_b200.tokenizer_manager import TokenizerManager
from oracle import cpu_oracle as O

pytestmark = pytest.mark.gpu

# "a".."d" join in every way the rules say; no rule touches "." and so it always stands alone
RULES = [[97, 98, 300], [300, 300, 301], [97, 97, 302], [301, 99, 70000], [99, 99, 4000000000], [70000, 302, 305], [98, 100, 306], [999, 97, 307],
         [307, 98, 308], [302, 302, 309], [97, 98, 310], [4000000000, 309, 311], [306, 97, 312]]


def _text(rng, lengths, n):
    parts, size = [], 0
    while size < n:
        parts.append(rng.integers(97, 101, int(rng.choice(lengths)), dtype=np.uint8))
        parts.append(np.array([46], np.uint8))
        size += parts[-2].size + 1
    return np.concatenate(parts)[:n]


@pytest.mark.parametrize("lengths", [[1, 2, 3, 7], [31, 32, 33], [1, 64, 200], [510, 511, 512, 513], [5, 1024], [3, 1600], [5000]])
@pytest.mark.parametrize("n", [1, 2, 1023, 1024, 1025, 1537, 2048, 40_007])
def test_segments_against_oracle(engine, lengths, n):
    data = _text(np.random.default_rng(n * 31 + lengths[-1]), lengths, n)
    tm = TokenizerManager(engine, {"merges": RULES})
    assert np.array_equal(tm.encodeBytes(data), O.replay_encode(data, RULES))
    applied = sum(not np.array_equal(O.replay_encode(data, RULES[:r + 1]), O.replay_encode(data, RULES[:r])) for r in range(len(RULES)))
    assert tm.lastRounds() == applied
    tm.destroy()


def test_a_handle_takes_texts_with_and_without_long_segments_in_turn(engine):
    rng = np.random.default_rng(3)
    tm = TokenizerManager(engine, {"merges": RULES})
    for lengths, n in (([4], 5000), ([4, 3000], 30_000), ([4], 90_001), ([40], 70)):
        data = _text(rng, lengths, n)
        assert np.array_equal(tm.encodeBytes(data), O.replay_encode(data, RULES))
    tm.destroy()


@pytest.mark.parametrize("length", [33, 34, 63, 64, 65, 95, 96, 97, 500, 1000, 1400, 1535])
@pytest.mark.parametrize("kind", ["a", "ab", "aab", "two letters", "runs"])
def test_long_segments_of_few_letters(engine, length, kind):
    """Pairs of equal tokens in runs either side of a warp's 32 tokens, whose every other one is taken, from the left; several of them a tile."""
    rng = np.random.default_rng(length)
    rules = [[97, 97, 300], [300, 300, 301], [301, 301, 302], [97, 98, 303], [303, 303, 304], [98, 98, 305], [305, 305, 306], [300, 98, 307],
             [98, 300, 308], [304, 304, 309], [302, 97, 310], [309, 97, 311], [305, 97, 312], [306, 306, 313], [302, 302, 314]]
    parts = []
    for k in range(12):
        m = max(1, length - int(rng.integers(0, 3)) if k % 3 else length)
        if kind == "two letters":
            w = 97 + rng.integers(0, 2, m)
        elif kind == "runs":
            w = np.concatenate([np.full(int(rng.integers(1, 80)), 97 + k % 2 if rng.random() < 0.8 else 98) for _ in range(m)])[:m]
        else:
            w = np.resize(np.frombuffer(kind.encode(), np.uint8), m)
        parts += [w.astype(np.uint8), np.full(int(rng.integers(1, 40)), 46, np.uint8)]
    for data in (np.concatenate(parts), parts[0], np.concatenate(parts[:3])):
        for use in (rules, rules[:1], rules[:4]):
            tm = TokenizerManager(engine, {"merges": use})
            assert np.array_equal(tm.encodeBytes(data), O.replay_encode(data, use)), (len(use), data.size)
            tm.destroy()
