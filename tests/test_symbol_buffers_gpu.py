"""Training on the symbol buffers (k_pair_count, k_argmax_setup, k_merge_compact, the tail fix-up of "literal" runs), which sharded runs
and the texts that no dictionary takes go through: the cases written for the edges of its tiles, batches and tables, with the
dictionary switched off, and a look at which of the two paths a run took."""
import numpy as np
import pytest

from gpu_bpe_b200 import TrainerSession, _lib
from oracle import cpu_oracle as O
from tests.helpers import small_text
from tests.test_train_gpu import (  # noqa: F401 (collected here, with the flag that the fixture below adds)
    test_batch_edges, test_early_stop_when_best_count_drops_below_two, test_graph_and_plain_launches_agree, test_heuristic_boundaries_on_device,
    test_id_exhaustion, test_incremental_with_frequent_equal_symbol_merges, test_incrementally_maintained_table_stays_exact, test_known_answers,
    test_literal_limit_at_every_alignment, test_long_run_candidate_list_and_batch_ends, test_pair_counts_exact, test_random_symbols_match_oracle,
    test_runs_of_equal_symbols, test_small_table_grows, test_text_corpus_matches_oracle)

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def on_symbol_buffers(monkeypatch):
    plain, destroy = TrainerSession._opts, TrainerSession.destroy

    def opts(*args, **kw):
        o = plain(*args, **kw)
        o.flags |= _lib.FLAG_SYMBOL_BUFFERS
        return o

    def checked(self):
        taken = self._h is not None and self.word_stats()
        destroy(self)
        assert not taken or taken["positions"] == taken["launches"] == 0
    monkeypatch.setattr(TrainerSession, "_opts", staticmethod(opts))
    monkeypatch.setattr(TrainerSession, "destroy", checked)
    yield
    monkeypatch.undo()


def test_which_path(engine, monkeypatch):
    data, mask, sym = small_text(2, 51, 120_000)
    want = O.train(sym, 260, "literal", threads=4)["merges"].tolist()
    monkeypatch.undo()                                     # (the plain options and destroy)
    launches = {}
    for flags in (0, _lib.FLAG_SYMBOL_BUFFERS, _lib.FLAG_SYMBOL_BUFFERS | _lib.FLAG_NO_GRAPH):
        s = TrainerSession.create(engine, data, mask, target_vocab_size=256 + 260, flags=flags)
        before = s.launches()
        m, c, _ = s.run()
        assert np.concatenate([m, c[:, None]], axis=1).tolist() == want
        launches[flags] = s.launches() - before
        assert (s.word_stats()["positions"] > 0) == (flags == 0)
        s.destroy()
    assert launches[0] < 20 and all(n >= 3 * 260 for f, n in launches.items() if f)
