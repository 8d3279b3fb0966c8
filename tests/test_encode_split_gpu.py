"""The walk that is split at every 32 bytes, where it can go wrong, against the CPU oracle: texts whose walks never meet, tokens longer
than a block and than the reach of a walk, chunk sizes either side of a block, of a tile and of what the walk takes, many short
documents, and inputs either side of the rule that chooses it."""
import numpy as np
import pytest

from gpu_bpe_b200 import TrieTokenizer, _lib, compileVocabToTrie
from oracle import cpu_oracle as O
from tests.helpers import small_text

pytestmark = pytest.mark.gpu

BYTES = [bytes([i]) for i in range(256)]
# runs of a: walks from different places keep their phase; long tokens: a walk jumps over whole blocks
RUNS = BYTES + [b"a" * k for k in (2, 3, 5, 7)] + [b"ab" * k for k in (1, 2, 16, 17, 48, 49)] + [b"abc" * 40, b"b" * 31, b"b" * 32, b"b" * 33, b"b" * 97]


def _runs(rng, n):
    parts, size = [], 0
    while size < n:
        unit = [b"a", b"ab", b"abc", b"b", b"xyz", b" "][rng.integers(6)]
        parts.append(np.frombuffer(unit * int(rng.integers(1, 200)), np.uint8))
        size += parts[-1].size
    return np.concatenate(parts)[:n]


@pytest.mark.parametrize("layout", ["auto", "hybrid"])
@pytest.mark.parametrize("chunk", [1, 31, 32, 33, 64, 512, 700, 2048, 16384, 16416])
@pytest.mark.parametrize("n", [1, 31, 33, 5000, 100_001])
def test_runs_and_long_tokens(engine, layout, chunk, n):
    data = _runs(np.random.default_rng(n + chunk), n)
    tok = TrieTokenizer(engine, compileVocabToTrie(RUNS), RUNS, {"layout": layout, "chunkSize": chunk})
    assert np.array_equal(tok.encodeBytes(data), O.encode(data, compileVocabToTrie(RUNS), chunk))
    tok.destroy()


@pytest.mark.parametrize("layout", ["auto", "hybrid"])
@pytest.mark.parametrize("docs", [1, 2, 31, 33, 3000])
def test_documents(engine, layout, docs):
    rng = np.random.default_rng(docs)
    data, _, sym = small_text(2, 19, 300_000)
    merges = O.train(sym, 400, "fixed", threads=4)["merges"].tolist()
    vocab = list(BYTES)
    for a, b, _, _ in merges:
        vocab.append(vocab[a] + vocab[b])
    offs = np.sort(np.concatenate([[0, data.size], rng.integers(0, data.size + 1, docs - 1)])).astype(np.uint64)
    trie = compileVocabToTrie(vocab)
    tok = TrieTokenizer(engine, trie, vocab, {"layout": layout})
    got, toff = tok.encodeBatch(data, offs)
    want, woff = O.encode_batch(data, offs, trie, tok.chunkSize)
    assert np.array_equal(got, want) and np.array_equal(toff, woff)
    tok.destroy()


def test_a_text_without_room_for_its_tokens(engine):
    data = _runs(np.random.default_rng(1), 9000)
    tok = TrieTokenizer(engine, compileVocabToTrie(RUNS), RUNS)
    want = O.encode(data, compileVocabToTrie(RUNS), tok.chunkSize)
    import ctypes as C
    out, n = np.full(want.size, 7, np.uint32), C.c_uint64()
    st = _lib.lib().b200bpe_encode(tok._h, data.ctypes.data, data.size, out.ctypes.data, want.size - 1, C.byref(n))
    assert _lib.STATUS[st] == "CAPACITY" and n.value == want.size and (out == 7).all()
    tok.destroy()


@pytest.mark.parametrize("n", [(38 << 20) - 5, 60 << 20])
@pytest.mark.parametrize("layout", ["auto", "hybrid"])
def test_both_sides_of_the_rule(engine, layout, n):
    """Large inputs, one chosen either way: the same tokens as in slices small enough for the split walk."""
    data = np.tile(_runs(np.random.default_rng(2), 1 << 20), 60)[:n]
    trie = compileVocabToTrie(RUNS)
    whole, sliced = (TrieTokenizer(engine, trie, RUNS, {"layout": layout, **o}) for o in ({}, {"encodeSliceBytes": 1 << 20}))
    assert np.array_equal(whole.encodeBytes(data), sliced.encodeBytes(data))
    whole.destroy(), sliced.destroy()


@pytest.mark.parametrize("layout", ["auto", "hybrid"])
def test_a_small_vocabulary_beside_a_large_one(engine, layout):
    """Handles whose tries ask for different amounts of shared memory, in every order of creation and use."""
    import torch
    data, _, sym = small_text(2, 23, 300_000)
    entries = list(BYTES)
    for a, b, _, _ in O.train(sym, 8000, "fixed", threads=8)["merges"].tolist():
        entries.append(entries[a] + entries[b])
    sizes = [8256, 320, 4096, 600, 2048]
    toks = [TrieTokenizer.fromVocab(engine, entries[:n], {"layout": layout}) for n in sizes]
    assert layout == "hybrid" or len({t.deviceLayout for t in toks if t.deviceLayout[0] == 2}) > 1
    large = np.tile(data, 200)               # beyond the split walk's range: the walk of whole chunks
    d_text, d_out = torch.from_numpy(data).cuda(), torch.empty(data.size, dtype=torch.int32, device="cuda")
    for t, n in 2 * list(zip(toks, sizes)):
        trie = compileVocabToTrie(entries[:n])
        want = O.encode(data, trie, t.chunkSize)
        assert np.array_equal(t.encodeBytes(data), want), n
        k = t.encodeDeviceNoAlloc(d_text.data_ptr(), data.size, d_out.data_ptr(), data.size)
        assert np.array_equal(d_out[:k].cpu().numpy().astype(np.uint32), want), n
        assert t.encodeBytes(large).size == O.encode(large, trie, t.chunkSize).size, n
    for t in toks:
        t.destroy()


@pytest.mark.parametrize("layout", ["auto", "hybrid"])
def test_one_handle_for_both_walks(engine, layout):
    """Sizes that go through either walk in turn on one handle, whose look-back descriptors grow with the tiles of the walk that runs."""
    data = np.tile(_runs(np.random.default_rng(5), 1 << 20), 60)
    trie = compileVocabToTrie(RUNS)
    one, sliced = (TrieTokenizer(engine, trie, RUNS, {"layout": layout, **o}) for o in ({}, {"encodeSliceBytes": 1 << 20}))
    for n in (60 << 20, 100, 5_000_001, 30 << 20, 60 << 20):
        assert np.array_equal(one.encodeBytes(data[:n]), sliced.encodeBytes(data[:n])), n
    fresh = TrieTokenizer(engine, trie, RUNS, {"layout": layout, "batchSliceBytes": 1 << 20})
    for docs in (40, 30_000, 7):              # slices of a batch that take different walks: few long documents, then many short ones
        offs = np.unique(np.concatenate([[0, 6 << 20, 12 << 20], (6 << 20) + np.arange(docs) * 200])).astype(np.uint64)
        got, toff = fresh.encodeBatch(data[:12 << 20], offs)
        want, woff = O.encode_batch(data[:12 << 20], offs, trie, fresh.chunkSize)
        assert np.array_equal(got, want) and np.array_equal(toff, woff), docs
    for t in (one, sliced, fresh):
        t.destroy()
