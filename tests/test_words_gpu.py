"""Training on the dictionary of distinct words ("fixed" compaction on one GPU) at the sizes where its kernels can go wrong:
word lengths either side of the short-word key (15 bytes), of the length field of the long-word table (255) and of the longest word
a dictionary takes (4,096), words across the edges of the 4,096-byte tiles, and a pair table that has to grow in mid-run.  The
oracle is the pass-by-pass CPU restatement; results are whole numbers and must be equal."""
import numpy as np
import pytest

from gpu_bpe_b200 import TrainerSession
from oracle import cpu_oracle as O

pytestmark = pytest.mark.gpu


def _check(engine, data, mask, merges, **kw):
    sym = data.astype(np.uint32) | (mask.astype(np.uint32) << 16)
    want = O.train(sym, merges, "fixed", threads=4)
    s = TrainerSession.create(engine, data, mask, target_vocab_size=256 + merges, compat_mode="fixed", **kw)
    assert np.array_equal(s.symbols(), sym)
    m, c, early = s.run()
    final = s.symbols().copy()
    table = {((k >> 32) << 16) | (k & 0xFFFF): v for k, v in s.pair_counts().items()}
    s.destroy()
    assert np.concatenate([m, c[:, None]], axis=1).tolist() == want["merges"].tolist()
    assert early == want["early_stop"] and np.array_equal(final, want["symbols"])
    assert table == O.pair_counts(final)


@pytest.mark.parametrize("length", [1, 2, 14, 15, 16, 17, 31, 254, 255, 256, 300, 4095, 4096, 4097, 9000])
def test_word_lengths(engine, length):
    """A few distinct words of one length, repeated in random order at every alignment (shorter words in between)."""
    rng = np.random.default_rng(length)
    words = [rng.integers(97, 101, size=length).astype(np.uint8) for _ in range(3)]
    words.append(words[0].copy())
    words[-1][-1] ^= 1                                   # differs from another word in its last byte only
    words += [words[1][:max(1, length - 1)], np.concatenate([words[1], words[1][:1]])]   # a prefix and an extension
    parts, starts, at = [], [], 0
    for _ in range(max(12, min(4000, 60_000 // length))):
        w = words[rng.integers(len(words))] if rng.random() < 0.7 else rng.integers(97, 100, size=rng.integers(1, 6)).astype(np.uint8)
        parts.append(w)
        starts.append(at)
        at += w.size
    data = np.concatenate(parts)
    mask = np.zeros(data.size, np.uint8)
    mask[starts] = 1
    _check(engine, data, mask, 60)


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 4095, 4096, 4097, 8191, 8192, 8193, 70_001])
def test_text_sizes_and_zero_bytes(engine, n):
    rng = np.random.default_rng(n)
    data = rng.integers(97, 103, size=n).astype(np.uint8)
    data[rng.random(n) < 0.02] = 0                       # a symbol 0 never pairs
    mask = (rng.random(n) < 0.18).astype(np.uint8)
    mask[0] = n % 2                                      # the first word starts at the first byte, marked or not
    _check(engine, data, mask, 40)


@pytest.mark.parametrize("log2", [4, 9, 12])
def test_pair_table_grows_in_mid_run(engine, log2):
    rng = np.random.default_rng(log2)
    n = 60_000
    data = (97 + np.minimum(rng.geometric(0.15, size=n), 25)).astype(np.uint8)
    mask = (rng.random(n) < 0.2).astype(np.uint8)
    _check(engine, data, mask, 700, table_log2=log2)
