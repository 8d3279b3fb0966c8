"""Device inputs of a trainer belong to the caller: they are read while create and reset run, and at no other time."""
import numpy as np
import pytest

from gpu_bpe_b200 import TrainerSession
from oracle import cpu_oracle as O
from tests.helpers import small_text

pytestmark = pytest.mark.gpu


def _runs(n):
    """Words of few letters: counts so large that a "literal" run reaches past its tail and starts again from the text."""
    rng = np.random.default_rng(n)
    data = (97 + rng.integers(0, 3, n)).astype(np.uint8)
    mask = (rng.random(n) < 0.18).astype(np.uint8)
    mask[0] = 1
    return data, mask


@pytest.mark.parametrize("text", ["words", "few letters", "a long word"])
@pytest.mark.parametrize("with_mask", [True, False])
@pytest.mark.parametrize("mode", ["literal", "fixed"])
def test_buffers_overwritten_after_create_and_reset(engine, text, with_mask, mode):
    import torch
    n = 70_001
    data, mask = _runs(n) if text == "few letters" else small_text(2, 31, n)[:2]
    if text == "a long word":
        data, mask = data.copy(), mask.copy()
        data[1000:9000] = 97
        mask[1000:9000] = 0
        mask[1000] = 1
    other = np.random.default_rng(1).integers(32, 127, n).astype(np.uint8)
    d_bytes, d_mask = torch.from_numpy(data.copy()).cuda(), torch.from_numpy(mask.copy()).cuda()
    s = TrainerSession.create(engine, d_bytes.data_ptr(), d_mask.data_ptr() if with_mask else None, n=n, device_pointers=True,
                              target_vocab_size=256 + 50, compat_mode=mode)
    for text in (data, other):
        sym = text.astype(np.uint32) | (mask.astype(np.uint32) << 16) if with_mask else O.word_boundary(text)
        want = O.train(sym, 50, mode, threads=4)
        d_bytes.fill_(0x78)
        d_mask.fill_(1)
        torch.cuda.synchronize()
        assert np.array_equal(s.symbols(), sym)
        m, c, early = s.run()
        assert np.concatenate([m, c[:, None]], axis=1).tolist() == want["merges"].tolist() and early == want["early_stop"]
        assert np.array_equal(s.symbols(), want["symbols"])
        # what the buffers hold at a reset is what the run after it works on
        d_bytes.copy_(torch.from_numpy(other))
        d_mask.copy_(torch.from_numpy(mask))
        torch.cuda.synchronize()
        s.reset()
    del d_bytes, d_mask
    s.destroy()
