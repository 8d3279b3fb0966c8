"""Texts that the dictionary of distinct words does not take, or cannot finish: what belongs to it is given back before the symbol
buffers are allocated, and a text of the trainer's own is not tried again at a reset."""
import numpy as np
import pytest

from gpu_bpe_b200 import BPEEngine, TrainerSession
from oracle import cpu_oracle as O

pytestmark = pytest.mark.gpu


def _one_word(n):
    """A word longer than a dictionary takes, then short ones."""
    rng = np.random.default_rng(n)
    data = (97 + rng.integers(0, 6, n)).astype(np.uint8)
    mask = (rng.random(n) < 0.2).astype(np.uint8)
    mask[:5000] = 0
    mask[0] = 1
    return data, mask


def _few_letters(n):
    """Counts so large that a "literal" run reaches past any tail."""
    rng = np.random.default_rng(n)
    data = (97 + rng.integers(0, 2, n)).astype(np.uint8)
    return data, (rng.random(n) < 0.1).astype(np.uint8)


@pytest.mark.parametrize("text,mode", [(_one_word, "fixed"), (_one_word, "literal"), (_few_letters, "literal")])
def test_reset_does_not_try_again(engine, text, mode):
    data, mask = text(60_000)
    want = O.train(data.astype(np.uint32) | (mask.astype(np.uint32) << 16), 30, mode, threads=4)
    s = TrainerSession.create(engine, data, mask, target_vocab_size=256 + 30, compat_mode=mode)
    for k in range(3):
        m, c, early = s.run()
        assert np.concatenate([m, c[:, None]], axis=1).tolist() == want["merges"].tolist() and early == want["early_stop"]
        assert np.array_equal(s.symbols(), want["symbols"])
        before = s.launches()
        s.reset()
        assert s.launches() - before == 1, "a reset of the symbol buffers tags the symbols and launches nothing else"
    s.destroy()


@pytest.mark.parametrize("device_pointers", [False, True])
def test_memory_for_the_symbol_buffers_only(device_pointers):
    """As much free memory as the symbol buffers need, and little more: the dictionary's tables (0.9 GB) do not fit beside them."""
    import torch
    n = 256 << 20
    rng = np.random.default_rng(3)
    data = (97 + rng.integers(0, 6, n, dtype=np.uint8)).astype(np.uint8)
    mask = (rng.integers(0, 8, n, dtype=np.uint8) == 0).astype(np.uint8)
    mask[:5000] = 0
    d_data, d_mask = torch.from_numpy(data).cuda(), torch.from_numpy(mask).cuda()
    args = ((d_data.data_ptr(), d_mask.data_ptr()) if device_pointers else (data, mask))
    lists = []
    for short in (False, True):
        e = BPEEngine(0).init()
        hold = None
        if short:
            torch.cuda.empty_cache()
            own = 0 if device_pointers else 2 * n
            room = 12 * n + own + (400 << 20)
            hold = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
        s = TrainerSession.create(e, *args, n=n, device_pointers=device_pointers, target_vocab_size=256 + 3, compat_mode="fixed")
        m, c, _ = s.run()
        lists.append(np.concatenate([m, c[:, None]], axis=1).tolist())
        s.destroy()
        e.destroy()
        del hold
        torch.cuda.empty_cache()
    assert lists[0] == lists[1] and len(lists[0]) == 3
