"""The device's answer to "is this text surely in NFC?": a normalising PreTokenizer gives the same bytes and word starts with the
device as without, whatever the text, and texts that need no normalising are recognised."""
import ctypes as C
import unicodedata

import numpy as np
import pytest

from gpu_bpe_b200 import PreTokenizer, _lib

pytestmark = pytest.mark.gpu

PLAIN = "plain ASCII, d\u00e9j\u00e0 vu, \u4f60\u597d \ud55c\uad6d\uc5b4 \u0440\u0443\u0441 \U0001F600 \u0627\u0644 1234\n"


def surely(engine, raw: bytes) -> int:
    a = np.frombuffer(raw, np.uint8)
    mask, f = np.empty(a.size, np.uint8), C.c_uint32()
    _lib.check(_lib.lib().b200bpe_pretokenize_gpu_nfc(engine.ctx, a.ctypes.data, a.size, mask.ctypes.data, C.byref(f)))
    return f.value


@pytest.mark.parametrize("middle", ["", "e\u0301", "\u1112\u1161\u11ab", "\u212b", "\u0958", "a\u0327\u0301", "\u0344", "\u2adc", "\u0378", "\u3099", "\U00011099\U000110ba"])
@pytest.mark.parametrize("before", [0, 4093, 9000])
def test_same_as_without_the_device(engine, middle, before):
    raw = ("x" * before + middle + PLAIN).encode()
    host, dev = PreTokenizer().preTokenizeBytes(raw), PreTokenizer(engine=engine).preTokenizeBytes(raw)
    assert np.array_equal(host["bytes"], dev["bytes"]) and np.array_equal(host["wordStarts"], dev["wordStarts"])
    assert surely(engine, raw) == (1 if middle == "" else 0)


@pytest.mark.parametrize("raw", [b"ab\xc3", b"ab\xc0\x80cd", b"\xe0\x80\x80 a", b"\xed\xa0\x80 a", b"\xf4\x90\x80\x80 a"])
def test_loosely_formed_bytes_are_taken_as_they_are(engine, raw):
    assert surely(engine, raw) == 0
    dev, plain = PreTokenizer(engine=engine).preTokenizeBytes(raw), PreTokenizer(normalize=False, engine=engine).preTokenizeBytes(raw)
    assert dev["bytes"].tobytes() == raw and np.array_equal(dev["wordStarts"], plain["wordStarts"])


def test_malformed_bytes_are_still_refused(engine):
    with pytest.raises(ValueError):
        PreTokenizer(engine=engine).preTokenizeBytes(b"a\x80b")


def test_every_code_point_called_plain_is_left_alone(engine):
    """All code points in blocks: where the device says yes, Python agrees that nothing in the block can matter to NFC."""
    for lo in range(0, 0x110000, 0x100):
        text = "".join(chr(c) for c in range(lo, lo + 0x100) if not 0xD800 <= c < 0xE000)
        if text and surely(engine, text.encode()):
            assert unicodedata.is_normalized("NFC", text), hex(lo)
            assert not any(unicodedata.combining(c) for c in text), hex(lo)
