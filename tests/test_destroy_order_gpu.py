"""Handles outlive the engine that they were made with: what they hold goes back whichever is destroyed first."""
import numpy as np
import pytest

from gpu_bpe_b200 import BPEEngine, TrainerSession, TrieTokenizer
from gpu_bpe_b200.tokenizer import DECODE_ON_DEVICE
from oracle import cpu_oracle as O
from tests.helpers import small_text

pytestmark = pytest.mark.gpu


def test_engine_first():
    data, mask, sym = small_text(2, 61, 100_000)
    want = O.train(sym, 100, "literal", threads=4)["merges"].tolist()
    vocab = [bytes([i]) for i in range(256)] + [b"the ", b"ab"]
    tokens = np.random.default_rng(0).integers(0, 258, DECODE_ON_DEVICE, dtype=np.uint32)
    for _ in range(3):
        e = BPEEngine(0).init()
        sessions = [TrainerSession.create(e, data, mask, target_vocab_size=256 + 100) for _ in range(2)]
        tok = TrieTokenizer.fromVocab(e, vocab)
        text = tok.decode(tokens)
        assert text == b"".join(vocab[t] for t in tokens) and tok.encodeBytes(np.frombuffer(text, np.uint8)).size > 0
        m, c, _ = sessions[0].run()
        assert np.concatenate([m, c[:, None]], axis=1).tolist() == want
        e.destroy()
        e.destroy()
        assert tok.decode(tokens) == text                  # (the general way: the engine is gone)
        m, c, _ = sessions[1].run()
        assert np.concatenate([m, c[:, None]], axis=1).tolist() == want
        for h in (sessions[1], tok, sessions[0]):
            h.destroy()
