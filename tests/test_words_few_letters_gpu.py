"""Which texts of distinct words train on the dictionary: large ones of few letters go to the symbol buffers, by their letters, their
size, how often words repeat and how many merges are wanted; the merge lists are the oracle's on both."""
import numpy as np
import pytest

from gpu_bpe_b200 import TrainerSession, _lib
from oracle import cpu_oracle as O

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _lines(letters, n, again, width=65):
    """Lines of random letters behind a space, each distinct line `again` times."""
    rng = np.random.default_rng(letters * again + n)
    rows = n // width
    pool = rng.integers(65, 65 + letters, (-(-rows // again), width), dtype=np.uint8)
    text = np.tile(pool, (again, 1))[:rows]
    text[:, 0] = 32
    mask = np.zeros(text.shape, np.uint8)
    mask[:, 0] = 1
    return text.reshape(-1), mask.reshape(-1)


@pytest.mark.parametrize("letters,n,again,merges,mode,dictionary", [
    (4, 9 * MIB, 1, 40, "fixed", False),
    (4, 10 * MIB, 1, 40, "literal", False),
    (2, 10 * MIB, 1, 40, "literal", False),      # few enough pairs for the long tail
    (4, 7 * MIB, 1, 40, "fixed", True),          # small
    (4, 9 * MIB, 8, 40, "fixed", True),          # repeated words
    (64, 9 * MIB, 1, 40, "fixed", True),         # many letters
    (64, 10 * MIB, 1, 40, "literal", True),
    (4, 9 * MIB, 1, 4000, "fixed", True),        # enough later merges
])
def test_which_path(engine, letters, n, again, merges, mode, dictionary):
    data, mask = _lines(letters, n, again)
    want = O.train(data.astype(np.uint32) | (mask.astype(np.uint32) << 16), 4, mode, threads=4)["merges"].tolist()
    lists = []
    for flags in (0, _lib.FLAG_SYMBOL_BUFFERS):
        s = TrainerSession.create(engine, data, mask, target_vocab_size=256 + merges, compat_mode=mode, flags=flags)
        assert (s.word_stats()["positions"] > 0) == (dictionary and not flags)
        m, c, _ = s.run(40)
        lists.append(np.concatenate([m, c[:, None]], axis=1).tolist())
        s.destroy()
    assert lists[0] == lists[1] and lists[0][:4] == want


def test_columns_are_not_letters(engine):
    """A table whose columns are 64 bytes apart, two of them constant: the sample does not fall into one column."""
    rng = np.random.default_rng(1)
    text = rng.integers(33, 97, (9 * MIB // 64, 64), dtype=np.uint8)
    text[:, :3] = (32, 50, 48)
    mask = np.zeros(text.shape, np.uint8)
    mask[:, 0] = 1
    s = TrainerSession.create(engine, text.reshape(-1), mask.reshape(-1), target_vocab_size=256 + 10, compat_mode="fixed")
    assert s.word_stats()["positions"] > 0
    s.destroy()


def test_runs_of_equal_letters_do_not_count(engine):
    """Nearly every pair is of two equal bytes, and the runs are gone with a merge each."""
    data, mask = _lines(64, 9 * MIB, 1)
    rows = data.reshape(-1, 65)
    rows[:, 9:] = 65
    s = TrainerSession.create(engine, data, mask, target_vocab_size=256 + 10, compat_mode="fixed")
    assert s.word_stats()["positions"] > 0
    s.destroy()
