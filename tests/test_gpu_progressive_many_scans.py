"""A progressive frame of many scans: they are decoded in groups, in order, and
the memory they take does not grow with their number."""
import struct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def seg(m, body):
    return bytes([0xFF, m]) + struct.pack(">H", len(body) + 2) + body


def frame(scans):
    """8x8 grey: a DC scan, then AC scans that each set coefficient 1 to +-1 (the last one stands)."""
    dht = seg(0xC4, bytes([0x00, 1] + [0] * 15 + [0])) + seg(0xC4, bytes([0x10, 1, 1] + [0] * 14 + [0x01, 0x00]))
    head = b"\xff\xd8" + seg(0xDB, b"\0" + b"\x20" * 64) + seg(0xC2, struct.pack(">BHHB", 8, 8, 8, 1) + bytes([1, 0x11, 0]))
    body = b"".join(seg(0xDA, bytes([1, 1, 0, 1, 63, 0])) + bytes([0b01100000 if up else 0b00100000]) for up in scans)
    return head + dht + seg(0xDA, bytes([1, 1, 0, 0, 0, 0])) + b"\0" + body + b"\xff\xd9"


@pytest.mark.parametrize("n", [62, 63, 64, 65, 127, 200])
def test_scans_in_groups(cj, oracle_mod, n):
    for last in (True, False):
        data = frame([k % 2 == 0 for k in range(n - 1)] + [last])
        with cj.Reader() as r:
            r.open_bytes(data)
            assert np.array_equal(r.pixels(), oracle_mod.decode(data).pixels)


def test_memory_does_not_grow_with_the_scans(cj, oracle_mod):
    import torch

    few, many = frame([True] * 3), frame([k % 3 == 0 for k in range(19999)] + [True])
    want = oracle_mod.decode(few).pixels
    with cj.Reader() as r:
        r.open_bytes(few)
        free = torch.cuda.mem_get_info()[0]
        r.open_bytes(many)
        assert np.array_equal(r.pixels(), want)
        assert free - torch.cuda.mem_get_info()[0] < 16 << 20
