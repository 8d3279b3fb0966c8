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
