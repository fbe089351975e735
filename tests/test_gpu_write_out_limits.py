"""A restart interval whose data hold more blocks than 26 bits count, in front
of a regular one: the decode of the interval behind it stores inside the image."""
import struct

import numpy as np
import pytest

from cudajpeg_b200 import workloads as W

pytestmark = pytest.mark.gpu


def overlong_interval_file():
    """16x8 grey, an interval per MCU; DC and AC codes of one bit ('0': no
    difference, end of block), so the first interval's zeros are 2-bit blocks."""
    def seg(m, body):
        return bytes([0xFF, m]) + struct.pack(">H", len(body) + 2) + body

    def dht(cls, symbols):
        return bytes([cls << 4, 2] + [0] * 15) + bytes(symbols)

    zeros = ((1 << 26) + (1 << 22)) * 2 // 8
    return (b"\xff\xd8" + seg(0xDB, b"\0" + b"\1" * 64) + seg(0xC0, struct.pack(">BHHB", 8, 8, 16, 1) + bytes([1, 0x11, 0]))
            + seg(0xC4, dht(0, [0, 1])) + seg(0xC4, dht(1, [0, 1])) + seg(0xDD, struct.pack(">H", 1))
            + seg(0xDA, bytes([1, 1, 0, 0, 63, 0])) + b"\0" * zeros + b"\xff\xd0" + b"\0" + b"\xff\xd9")


def test_interval_of_more_than_2_26_blocks(cj, oracle_mod):
    data = overlong_interval_file()
    good = W.small_case(5, 200, 136, "420", 80, 3).data
    want = oracle_mod.decode(good).pixels
    with cj.Reader() as r:
        assert r.open_bytes(data, check=False) == cj.SYNTAX_ERROR
        r.open_bytes(good)
        assert np.array_equal(r.pixels(), want)
    with cj.Batch() as b:
        imgs, errs = b.decode([good, data, good])
        assert list(errs) == [0, cj.SYNTAX_ERROR, 0]
        assert np.array_equal(imgs[0], want) and np.array_equal(imgs[2], want)
