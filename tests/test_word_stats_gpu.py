"""Statistics of a run name the kernels that ran: the dictionary's merge kernel, or those of the symbol buffers."""
import numpy as np
import pytest

from gpu_bpe_b200 import TrainerSession, _lib
from oracle import cpu_oracle as O
from tests.helpers import small_text

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["literal", "fixed"])
def test_dictionary(engine, mode):
    data, mask, sym = small_text(2, 17, 300_000)
    s = TrainerSession.create(engine, data, mask, target_vocab_size=256 + 300, compat_mode=mode, flags=_lib.FLAG_TIME_KERNELS)
    positions = sum(len(w) for w in {bytes(w) for w in np.split(data, np.flatnonzero(mask)[1:])})
    for _ in range(2):
        m, _, _ = s.run()
        ws, ks = s.word_stats(), s.kernel_stats()
        assert not any(ks.values())
        assert ws["merges"] == len(m) == 300 and ws["launches"] >= 3 and ws["merge_ms"] > 0
        assert ws["positions"] == positions if mode == "fixed" else 0 < ws["positions"] <= positions
        assert 0 < ws["list_entries"] <= 2 * ws["positions"] and ws["table_scans"] >= 1
        assert ws["bytes"] > 8 * ws["list_entries"]
        s.reset()
        assert s.word_stats()["launches"] == s.word_stats()["merges"] == 0
    s.destroy()


def test_symbol_buffers(engine):
    data, mask, sym = small_text(2, 18, 100_000)
    mask = mask.copy()
    mask[2000:9000] = 0                                   # a word longer than a dictionary takes
    s = TrainerSession.create(engine, data, mask, target_vocab_size=256 + 40, flags=_lib.FLAG_TIME_KERNELS)
    m, c, _ = s.run()
    ks = s.kernel_stats()
    assert not any(s.word_stats().values())
    assert ks["merge_compact_launches"] >= 40 and ks["merge_compact_ms"] > 0 and ks["merge_compact_bytes"] > 4 * 40 * data.size
    s.destroy()


def test_counts_without_room(engine):
    data, mask, sym = small_text(2, 19, 50_000)
    s = TrainerSession.create(engine, data, mask, target_vocab_size=300)
    want = O.pair_counts(sym)
    with pytest.raises(_lib.B200BPEError) as e:
        s.pair_counts(cap=10)
    assert e.value.status_name == "CAPACITY"
    assert len(s.pair_counts(cap=len(want))) == len(want)
    s.destroy()
