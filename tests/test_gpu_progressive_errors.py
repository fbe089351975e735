"""Malformed progressive scans: a restart interval ends at its first error, so a
value outside int16 (UNSUPPORTED_ERROR) is what a frame reports even where the
data behind it hold invalid codes (SYNTAX_ERROR) in the same block or in a block
with a lower index."""
import struct

import numpy as np
import pytest

from cudajpeg_b200 import workloads as W

pytestmark = pytest.mark.gpu


def seg(m, body):
    return bytes([0xFF, m]) + struct.pack(">H", len(body) + 2) + body


def bits(s):
    s = s.replace(" ", "")
    s += "0" * (-len(s) % 8)
    return bytes(int(s[k:k + 8], 2) for k in range(0, len(s), 8)).replace(b"\xff", b"\xff\x00")


def frame(w, h, luma, script):
    """4:2:0 (luma 0x22) or grey (0x11).  DC codes: 0 size 0, 10 size 11; AC codes: 0 EOB, 10 run 0 size 15,
    110 run 0 size 1; all others are invalid."""
    n = 3 if luma == 0x22 else 1
    comps = b"".join(bytes([c + 1, luma if c == 0 else 0x11, 0]) for c in range(n))
    out = b"\xff\xd8" + seg(0xDB, b"\0" + b"\x01" * 64) + seg(0xC2, struct.pack(">BHHB", 8, h, w, n) + comps)
    out += seg(0xC4, bytes([0x00, 1, 1] + [0] * 14 + [0, 11])) + seg(0xC4, bytes([0x10, 1, 1, 1] + [0] * 13 + [0, 15, 1]))
    for ss, se, al, data in script:
        out += seg(0xDA, bytes([1, 1, 0, ss, se, al])) + bits(data)
    return out + b"\xff\xd9"


BIG_AC = "10" + "1" * 15     # 32767 << 13
BIG_DC = "10" + "1" * 11     # 2047 << 13
CASES = {
    # the invalid code follows in the same block
    "same block": (8, 8, 0x11, [(0, 0, 0, "0"), (1, 63, 13, BIG_AC + "111")]),
    # luma blocks run through both MCUs (16 x 16 samples each) row by row: the third block (MCU 1, index 6) has the
    # value, the fifth (MCU 0, index 2) the invalid code
    "lower index, AC": (32, 16, 0x22, [(0, 0, 0, "0" * 8), (1, 63, 13, "0 0" + BIG_AC + "0 0 111")]),
    "lower index, DC": (32, 16, 0x22, [(0, 0, 13, "0 0" + BIG_DC + "0 11")]),
    # two values out of range
    "two values": (32, 16, 0x22, [(0, 0, 0, "0" * 8), (1, 63, 13, "0 0" + BIG_AC + "0 0" + BIG_AC + "0 0 0 0")]),
}
SYNTAX = {
    "code first": (8, 8, 0x11, [(0, 0, 0, "0"), (1, 63, 13, "111")]),
    "code first, DC": (32, 16, 0x22, [(0, 0, 13, "0 11" + BIG_DC)]),
    "code in an earlier block": (32, 16, 0x22, [(0, 0, 0, "0" * 8), (1, 63, 13, "0 111" + BIG_AC)]),
}


@pytest.mark.parametrize("name", list(CASES) + list(SYNTAX))
def test_first_error_of_an_interval(cj, oracle_mod, name):
    args, want = (CASES[name], cj.UNSUPPORTED_ERROR) if name in CASES else (SYNTAX[name], cj.SYNTAX_ERROR)
    data = frame(*args)
    good = W.small_case(2, 64, 48, "420").data
    with cj.Reader() as r:
        assert r.open_bytes(data, check=False) == want
        r.open_bytes(good)
        assert np.array_equal(r.pixels(), oracle_mod.decode(good).pixels)


def sof(w, h):
    return seg(0xC2, struct.pack(">BHHB", 8, h, w, 1) + bytes([1, 0x11, 0]))


DC = seg(0xDA, bytes([1, 1, 0, 0, 0, 0]))


@pytest.mark.parametrize("first,second,scan,ok", [((8, 8), (4096, 4096), True, False), ((8, 8), (4096, 4096), False, False),
                                                  ((64, 64), (8, 8), True, True), ((64, 64), (64, 64), True, True),
                                                  ((256, 8), (8, 256), True, False), ((256, 8), (8, 256), False, True)])
def test_a_second_frame_header_stays_inside_the_coefficients(cj, first, second, scan, ok):
    """The first scan sizes the coefficient buffer and its rows of blocks; later scans that do not fit it, and
    a larger last frame, are refused."""
    head = b"\xff\xd8" + seg(0xDB, b"\0" + b"\x01" * 64) + seg(0xC4, bytes([0x00, 1, 1] + [0] * 14 + [0, 11]))
    zeros = bytes(-(-(first[0] // 8) * (first[1] // 8) // 8))
    data = head + sof(*first) + DC + zeros + sof(*second) + ((DC + bytes(32768)) if scan else seg(0xFE, b"comment")) + b"\xff\xd9"
    with cj.Reader(host_coefficients=True) as r:
        assert r.open_bytes(data, check=False) == (0 if ok else cj.SYNTAX_ERROR)
        if ok:
            assert (r.pixels() == 128).all() and r.pixels().shape[:2] == (second[1], second[0])
            assert not r.coefficients()[0].any()
        good = W.small_case(2, 64, 48, "420").data
        r.open_bytes(good)
