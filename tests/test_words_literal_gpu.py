""""literal" compaction on the dictionary of distinct words plus the symbols of the text's tail, against the pass-by-pass oracle: merge
list, counts, the live symbols (older contents included) and the pair table after runs of every length; tails of one warp row and
of many; pairs of equal symbols; tails that a merge reaches past (the symbol buffers then take the run); pair tables that grow."""
import numpy as np
import pytest

from gpu_bpe_b200 import TrainerSession
from oracle import cpu_oracle as O
from tests.helpers import small_text

pytestmark = pytest.mark.gpu


def _check(engine, data, mask, merges, **kw):
    sym = data.astype(np.uint32) | (mask.astype(np.uint32) << 16)
    s = TrainerSession.create(engine, data, mask, target_vocab_size=256 + max(merges), compat_mode="literal", **kw)
    done, got = 0, []
    for upto in merges:                                  # the state between calls, and after the last
        m, c, early = s.run(upto - done)
        got += np.concatenate([m, c[:, None]], axis=1).tolist() if len(m) else []
        done = upto
        want = O.train(sym, upto, "literal", threads=4)
        assert got == want["merges"].tolist() and early == want["early_stop"]
        final = s.symbols().copy()
        assert np.array_equal(final, want["symbols"])
        table = {((k >> 32) << 16) | (k & 0xFFFF): v for k, v in s.pair_counts().items()}
        assert table == O.pair_counts(final)
        if early:
            break
    s.destroy()


@pytest.mark.parametrize("kind", [1, 2, 5])
@pytest.mark.parametrize("n", [1200, 30_000, 131_071, 1_000_003])
def test_texts(engine, kind, n):
    data, mask, _ = small_text(kind, 60 + kind, n)
    _check(engine, data, mask, [1, 2, 3, 5, 40, 150] if n < 1_000_000 else [1, 2, 300])


@pytest.mark.parametrize("n", [5, 64, 257, 4097, 70_001])
@pytest.mark.parametrize("alphabet", [2, 5, 40])
def test_random_bytes(engine, n, alphabet):
    """Small alphabets: counts so large that the tail is soon used up, and runs of equal symbols."""
    rng = np.random.default_rng(n + alphabet)
    data = (97 + rng.integers(0, alphabet, n)).astype(np.uint8)
    data[rng.random(n) < 0.02] = 0
    mask = (rng.random(n) < 0.18).astype(np.uint8)
    _check(engine, data, mask, [1, 2, 3, 60])


@pytest.mark.parametrize("length", [3, 40, 300])
def test_runs_across_the_limit(engine, length):
    """Words of one repeated letter, so that runs of dropped symbols lie across the limit and the end of the copied part."""
    rng = np.random.default_rng(length)
    words = [np.full(int(rng.integers(1, length + 1)), 97 + int(rng.integers(0, 30)), np.uint8) for _ in range(60_000 // length)]
    data = np.concatenate(words)
    mask = np.zeros(data.size, np.uint8)
    mask[np.cumsum([0] + [w.size for w in words[:-1]])] = 1
    _check(engine, data, mask, [1, 2, 3, 4, 5, 6, 50])


def test_pair_table_grows(engine):
    data, mask, _ = small_text(2, 77, 200_000)
    _check(engine, data, mask, [64, 500], table_log2=9)
