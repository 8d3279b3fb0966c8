"""Decoding from several threads on one tokenizer, the decoder's C entry points, and which calls go to the device at all: a streaming
server decodes a few tokens at a time from its worker threads."""
import ctypes as C
import threading

import numpy as np
import pytest

from gpu_bpe_b200 import BPEEngine, TrainerSession, TrieTokenizer, _lib
from gpu_bpe_b200.tokenizer import DECODE_ON_DEVICE
from tests.helpers import small_text
from tests.test_decode_gpu import VOCAB, _loop

pytestmark = pytest.mark.gpu


def _together(work, n):
    """Runs work(0..n-1) in n threads that start at once; re-raises what one of them raised."""
    failed, start = [], threading.Barrier(n)

    def one(i):
        try:
            start.wait(60)
            work(i)
        except BaseException as e:
            failed.append(e)
    threads = [threading.Thread(target=one, args=(i,)) for i in range(n)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not any(t.is_alive() for t in threads)
    if failed:
        raise failed[0]


def test_several_threads_on_one_tokenizer(engine):
    tok = TrieTokenizer.fromVocab(engine, list(VOCAB))

    def work(i):
        rng = np.random.default_rng(i)
        for k in range(40):
            n = int(rng.choice([1, 50, DECODE_ON_DEVICE, 5000, 60_000]))
            tokens = rng.integers(0, [256, 260, 300][i % 3], n, dtype=np.uint32)
            assert tok.decode(tokens) == _loop(VOCAB, tokens), (i, k, n)
    _together(work, 6)
    tok.destroy()


def test_the_vocabulary_changes_and_a_trainer_runs_meanwhile(engine):
    """Entry 259 has one of two values at any time; another thread's run on the same engine records graphs on its stream."""
    vocab = list(VOCAB)
    tok = TrieTokenizer.fromVocab(engine, vocab)
    data, mask, _ = small_text(1, 5, 200_000)
    lists = []

    def work(i):
        if i == 0:
            for k in range(30):
                vocab[259] = [b"ab", b"longer"][k % 2]
                tok.decode(np.full(DECODE_ON_DEVICE, 97, np.uint32))
        elif i == 1:
            for _ in range(6):
                s = TrainerSession.create(engine, data, mask, target_vocab_size=256 + 300, flags=_lib.FLAG_FULL_RECOUNT)
                lists.append(s.run()[0].tolist())
                s.destroy()
        else:
            for k in range(60):
                got = tok.decode(np.full(DECODE_ON_DEVICE + 7 * k, 259, np.uint32))
                assert got in (b"ab" * (DECODE_ON_DEVICE + 7 * k), b"longer" * (DECODE_ON_DEVICE + 7 * k))
    _together(work, 4)
    assert all(m == lists[0] for m in lists) and len(lists[0]) == 300
    tok.destroy()


@pytest.mark.parametrize("n", [1, 3, 255, 1023, 1024, 1025, 2047, 4097])
@pytest.mark.parametrize("top", [256, 260, 300, 2**32])
def test_device_sizes(engine, n, top):
    """The device's way below the length from which it is taken."""
    tok = TrieTokenizer.fromVocab(engine, list(VOCAB))
    tokens = np.random.default_rng(n + top % 999).integers(0, top, n, dtype=np.uint32)
    assert tok._decode_on_device(tokens) == _loop(VOCAB, tokens)
    long = np.full(n, 257, np.uint32)            # more bytes than a first call expects
    assert tok._decode_on_device(long) == b"x" * (300 * n)
    tok.destroy()


def test_short_calls_stay_on_the_host(engine):
    tok = TrieTokenizer.fromVocab(engine, list(VOCAB))
    for n in (1, 10, 100, DECODE_ON_DEVICE - 1):
        tokens = np.random.default_rng(n).integers(0, 300, n, dtype=np.uint32)
        assert tok.decode(tokens) == _loop(VOCAB, tokens) and tok._dh is None
    tokens = np.random.default_rng(0).integers(0, 300, DECODE_ON_DEVICE, dtype=np.uint32)
    assert tok.decode(tokens) == _loop(VOCAB, tokens) and tok._dh is not None
    tok.destroy()


def test_c_entry_points():
    e = BPEEngine(0).init()
    L, h, n = _lib.lib(), C.c_void_p(), C.c_uint64()
    blob = np.frombuffer(b"".join(VOCAB), np.uint8)
    off = np.concatenate([[0], np.cumsum([len(v) for v in VOCAB])]).astype(np.uint64)
    assert L.b200bpe_decoder_create(e.ctx, blob.ctypes.data, off.ctypes.data, len(VOCAB), C.byref(h)) == 0
    tokens = np.array([256, 97, 999, 257], np.uint32)
    want = _loop(VOCAB, tokens)
    out = np.full(len(want), 7, np.uint8)
    status = lambda st: _lib.STATUS[st]
    assert status(L.b200bpe_decoder_decode(h, tokens.ctypes.data, 4, out.ctypes.data, out.size - 1, C.byref(n))) == "CAPACITY"
    assert n.value == len(want) and (out == 7).all()
    assert status(L.b200bpe_decoder_decode(h, tokens.ctypes.data, 4, None, 0, C.byref(n))) == "CAPACITY" and n.value == len(want)
    assert status(L.b200bpe_decoder_decode(h, tokens.ctypes.data, 4, out.ctypes.data, out.size, C.byref(n))) == "OK"
    assert out.tobytes() == want and n.value == len(want)
    assert status(L.b200bpe_decoder_decode(h, None, 0, None, 0, C.byref(n))) == "OK" and n.value == 0
    assert status(L.b200bpe_decoder_decode(h, None, 4, out.ctypes.data, out.size, C.byref(n))) == "BAD_ARG"
    for k in (4, 2, 0, 3):                          # in two steps; a second read gives the same text again
        assert status(L.b200bpe_decoder_run(h, tokens.ctypes.data, k, C.byref(n))) == "OK"
        want = _loop(VOCAB, tokens[:k])
        assert n.value == len(want)
        for _ in range(2):
            out = np.zeros(len(want) + 1, np.uint8)
            if k:
                assert status(L.b200bpe_decoder_read(h, out.ctypes.data, len(want) - 1)) == "CAPACITY"
            assert status(L.b200bpe_decoder_read(h, out.ctypes.data, out.size)) == "OK" and out[:-1].tobytes() == want
    L.b200bpe_decoder_destroy(h)
    e.destroy()
