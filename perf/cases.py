"""The work a user of this library has it do, as cases that can be timed: training a vocabulary, encoding with it
(prompts, files, batches of documents, on the host and on the device), decoding, the merge-replay encoder, and the
pre-tokeniser.

Corpora are the seeded synthetic text of gpu_bpe_b200/synth.py (kind 1 ASCII, 2 UTF-8 script mix, 5 heavy-tailed mix with
base64-like strings), the sizes those of the repository's own benchmark configurations and tests, cut down where a pass
would take longer than two seconds.  Encoding uses a vocabulary trained on other blocks of the same text ("near") or, as
benchmark configuration 4 does, on a text with other words ("far").  Everything is integers: results are exact.
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

from gpu_bpe_b200 import BPEEngine, BPETrainer, PreTokenizer, TrainerSession, TrieTokenizer, _lib, synth
from gpu_bpe_b200.tokenizer_manager import TokenizerManager

KIB, MIB = 1 << 10, 1 << 20
SPACE = 1 << 40              # length of the virtual corpus that near texts are blocks of
VOCAB_SEED, VOCAB_MERGES = 3, 32000
LARGEST = 256 * MIB          # bytes of the largest training and encoding inputs


def listed():
    return [
        # a chat prompt: one small encodeBytes call, latency only (the full 32,256-entry vocabulary of the benchmark)
        {"name": "encode_prompt", "op": "encode", "bytes": 2 * KIB, "vocab": 32256, "text": "near"},
        # a large file with the API's default vocabulary size (4,096), ordinary host memory, into the caller's buffer
        {"name": "encode_file", "op": "encode_into", "bytes": 4 * MIB + 13, "vocab": 4096, "text": "near", "pinned": False},
        # preparing a data set, documents in host memory (mean 4 KiB, as benchmark configuration 4; pinned, as bench.py has them)
        {"name": "encode_docs_host", "op": "encode_batch_into", "bytes": 64 * MIB, "docs": 16384, "vocab": 32256, "text": "far", "pinned": True},
        # the same with everything resident on the device: a quarter of benchmark configuration 4
        {"name": "encode_docs_device", "op": "encode_batch_device", "bytes": LARGEST, "docs": 65536, "vocab": 32256, "text": "far"},
        # the text of a stored token stream
        {"name": "decode", "op": "decode", "bytes": 256 * KIB, "vocab": 32256, "text": "near"},
        # the Tokenizer tab of the reference: merge rules replayed over a pasted document
        {"name": "replay_document", "op": "replay", "bytes": 192 * KIB + 7, "rules": 4000, "text": "near"},
        # word starts of a corpus before training, bytes in, mask out
        {"name": "pretokenize", "op": "pretokenize", "bytes": 32 * MIB, "kind": 2},
        # the smallest training call: a page of text without a pre-tokeniser (device heuristic), API defaults otherwise
        {"name": "train_page", "op": "train", "bytes": 64 * KIB, "kind": 1, "target": 512, "pretok": "none", "mode": "literal"},
        # benchmark configuration 1 through the public trainer: 1 MiB of ASCII, 1,000 merges
        {"name": "train_config1", "op": "train", "bytes": MIB, "kind": 1, "target": 1256, "pretok": "device", "mode": "literal"},
        # an ordinary corpus with the API's defaults (4,096 entries, mode as shipped), end to end from host bytes
        {"name": "train_default", "op": "train", "bytes": 24 * MIB + 5, "kind": 2, "target": 4096, "pretok": "device", "mode": "literal"},
        # benchmark configuration 2: 64 MiB, 8,000 merges, corpus resident on the device
        {"name": "train_config2", "op": "train_resident", "bytes": 64 * MIB, "kind": 2, "merges": 8000, "mode": "fixed"},
        # the largest: heavy-tailed text of benchmark configuration 5, resident
        {"name": "train_large", "op": "train_resident", "bytes": LARGEST, "kind": 5, "merges": 4000, "mode": "fixed"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["encode", "encode_into", "encode_batch_into", "encode_batch_device", "decode", "replay", "pretokenize", "train", "train",
                     "train_resident", "train_resident"])
    text = rng.choice(["near", "far"])
    if op == "encode":
        return {"op": op, "bytes": _log(rng, 64, 64 * KIB), "vocab": _log(rng, 512, 32256), "text": text}
    if op == "encode_into":
        return {"op": op, "bytes": _log(rng, 64 * KIB, 64 * MIB), "vocab": _log(rng, 512, 32256), "text": text, "pinned": rng.random() < 0.3}
    if op in ("encode_batch_into", "encode_batch_device"):
        n = _log(rng, 64 * KIB, 64 * MIB if op == "encode_batch_into" else LARGEST)
        c = {"op": op, "bytes": n, "docs": max(1, n // _log(rng, 256, 64 * KIB)), "vocab": _log(rng, 512, 32256), "text": text}
        return dict(c, pinned=rng.random() < 0.7) if op == "encode_batch_into" else c
    if op == "decode":
        return {"op": op, "bytes": _log(rng, KIB, MIB), "vocab": _log(rng, 512, 32256), "text": text}
    if op == "replay":
        return {"op": op, "bytes": _log(rng, KIB, MIB), "rules": _log(rng, 200, 16000), "text": text}
    if op == "pretokenize":
        return {"op": op, "bytes": _log(rng, 4 * KIB, 64 * MIB), "kind": rng.choice([1, 2, 5])}
    if op == "train":
        n = _log(rng, 32 * KIB, 32 * MIB)   # at least 128 bytes a merge: every run reaches its target
        return {"op": op, "bytes": n, "kind": rng.choice([1, 2, 5]), "target": _log(rng, 320, min(8192, 256 + n // 128)),
                "pretok": rng.choice(["device", "device", "none"]), "mode": rng.choice(["literal", "literal", "fixed"])}
    n = _log(rng, MIB, LARGEST)
    most = min(16000, n // 128, 4000 * LARGEST // n)
    return {"op": op, "bytes": n, "kind": rng.choice([1, 2, 5]), "merges": _log(rng, most // 8, most), "mode": rng.choice(["fixed", "literal"])}


@functools.lru_cache(None)
def _engine():
    return BPEEngine(0).init()


def _whole_characters(text):
    """Without the cut-off last character."""
    k = text.size
    while k and (text[k - 1] & 0xC0) == 0x80:
        k -= 1
    if k and text[k - 1] >= 0xC0:
        lead = int(text[k - 1])
        if k - 1 + (2 if lead < 0xE0 else 3 if lead < 0xF0 else 4) > text.size:
            return text[:k - 1]
    return text


def _text(case, seed):
    """`bytes` bytes of text: other blocks of the vocabulary's corpus, or text with other words."""
    block = (1 + (seed * 2654435761) % 900000) * MIB
    words = VOCAB_SEED if case["text"] == "near" else VOCAB_SEED + 1
    return synth.corpus_range(2, words, SPACE, block, case["bytes"])


@functools.lru_cache(None)
def _all_merges():
    """The merge list that the vocabularies are prefixes of, trained once."""
    data = synth.corpus_range(2, VOCAB_SEED, SPACE, 0, 16 * MIB)
    mask = PreTokenizer(normalize=False, engine=_engine()).preTokenizeBytes(_whole_characters(data))["wordStarts"]
    s = TrainerSession.create(_engine(), data[:mask.size], mask, target_vocab_size=256 + VOCAB_MERGES, compat_mode="fixed")
    merges, _, _ = s.run()
    s.destroy()
    return merges


@functools.lru_cache(None)
def _vocab(size):
    entries = [bytes([i]) for i in range(256)]
    for a, b, _ in _all_merges()[:size - 256].tolist():
        entries.append(entries[a] + entries[b])
    return entries


class _State:
    """Inputs and handles of one case; the handles are given back with it.  Encoders' outputs have room for a token a byte."""

    def __init__(self, case):
        self.case, self.handle = case, None

    def __del__(self):
        if self.handle is not None:
            self.handle.destroy()


def prepare(case, seed):
    s = _State(case)
    op, n, e = case["op"], case["bytes"], _engine()
    if "vocab" in case:
        s.handle = TrieTokenizer.fromVocab(e, _vocab(case["vocab"]))
        s.data = _text(case, seed)
        if "docs" in case:
            s.offsets = synth.doc_offsets(seed, n, case["docs"])
        if op == "decode":
            s.tokens = s.handle.encodeBytes(s.data)
        elif op == "encode_batch_device":
            s.d_text = torch.from_numpy(s.data).cuda()
            s.d_offsets = torch.from_numpy(s.offsets.view(np.int64)).cuda()
            s.d_tokens = torch.zeros(n, dtype=torch.int32, device="cuda")
            s.d_token_offsets = torch.zeros(case["docs"] + 1, dtype=torch.int64, device="cuda")
        else:
            s.tokens = np.zeros(n, np.uint32)
            if case.get("pinned"):
                s.pages = [torch.from_numpy(s.data).pin_memory(), torch.zeros(n, dtype=torch.int32).pin_memory()]
                s.data, s.tokens = s.pages[0].numpy(), s.pages[1].numpy().view(np.uint32)
            s.token_offsets = np.zeros(case.get("docs", 0) + 1, np.uint64)
    elif op == "replay":
        s.data = _text(case, seed)
        s.tokens = np.zeros(n, np.uint32)
        s.handle = TokenizerManager(e, {"merges": _all_merges()[:case["rules"]].tolist()})
    else:
        s.data = _whole_characters(synth.corpus(case["kind"], seed, n))
        if op == "train_resident":
            n = s.data.size
            s.d_bytes = torch.from_numpy(s.data).cuda()
            s.d_mask = torch.empty(n, dtype=torch.uint8, device="cuda")
            _lib.check(_lib.lib().b200bpe_pretokenize_device(e.ctx, C.c_void_p(s.d_bytes.data_ptr()), n, C.c_void_p(s.d_mask.data_ptr())))
            s.handle = TrainerSession.create(e, s.d_bytes.data_ptr(), s.d_mask.data_ptr(), n=n, device_pointers=True,
                                             target_vocab_size=256 + case["merges"], compat_mode=case["mode"])
        elif op == "pretokenize" or case["pretok"] == "device":
            s.pretok = PreTokenizer(engine=e)
        else:
            s.pretok = None
    return s


def run(s):
    case, op = s.case, s.case["op"]
    lib = _lib.lib()
    if op in ("encode", "replay"):
        ids = s.handle.encodeBytes(s.data)
        s.tokens[:ids.size] = ids
        return s.tokens, ids.size
    if op == "encode_into":
        count = C.c_uint64()
        _lib.check(lib.b200bpe_encode(s.handle._h, s.data.ctypes.data, s.data.size, s.tokens.ctypes.data, s.tokens.size, C.byref(count)))
        return s.tokens, count.value
    if op == "encode_batch_into":
        _lib.check(lib.b200bpe_encode_batch(s.handle._h, s.data.ctypes.data, s.offsets.ctypes.data, case["docs"], s.tokens.ctypes.data,
                                            s.tokens.size, s.token_offsets.ctypes.data))
        return s.tokens, s.token_offsets
    if op == "encode_batch_device":
        count = s.handle.encodeBatchDevice(s.d_text.data_ptr(), s.d_offsets.data_ptr(), case["docs"], case["bytes"], s.d_tokens.data_ptr(),
                                           s.d_tokens.numel(), s.d_token_offsets.data_ptr())
        return s.d_tokens, s.d_token_offsets, count
    if op == "decode":
        return np.frombuffer(s.handle.decode(s.tokens), np.uint8)
    if op == "pretokenize":
        r = s.pretok.preTokenizeBytes(s.data)
        return r["bytes"], r["wordStarts"]
    if op == "train":
        trainer = BPETrainer(_engine(), case["mode"])
        result = trainer.train(s.data, case["target"], s.pretok)
        return np.asarray(result["merges"], np.uint32), result["vocabSize"]
    s.handle.reset()
    return s.handle.run()


def work(case):
    """Every input byte read once, every result written once (about a token per 3 bytes; 12 bytes a merge)."""
    n, op = case["bytes"], case["op"]
    if op.startswith("encode"):
        return {"bytes": n + 4 * (n // 3) + 16 * case.get("docs", 0), "flops": 0}
    if op in ("decode", "replay"):
        return {"bytes": n + 4 * (n // 3), "flops": 0}
    if op == "pretokenize":
        return {"bytes": 2 * n, "flops": 0}
    merges = case["merges"] if op == "train_resident" else case["target"] - 256
    return {"bytes": (1 if case.get("pretok") else 2) * n + 12 * merges, "flops": 0}


def tolerance(case):
    return "exact"
