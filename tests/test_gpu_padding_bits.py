"""The bits that pad a restart interval to a byte: the standard wants ones, some
encoders write zeros, and a damaged file may hold any.  They are no part of a
block, so they never decide whether a file decodes, whatever the subsequence
size makes of them."""
import struct

import numpy as np
import pytest

from cudajpeg_b200 import workloads as W

pytestmark = pytest.mark.gpu


def repad(data, pad):
    """`data` (baseline, with restart markers) with `pad(interval, n)`'s low n bits as every interval's padding."""
    p, tables, restart, comps = 2, {}, 0, []
    while True:
        marker, n = data[p + 1], struct.unpack(">H", data[p + 2:p + 4])[0]
        seg = data[p + 4:p + 2 + n]
        if marker == 0xC4:
            q = 0
            while q < len(seg):
                counts, table, code, k = seg[q + 1:q + 17], {}, 0, q + 17
                for length in range(1, 17):
                    for _ in range(counts[length - 1]):
                        table[length, code] = seg[k]
                        code, k = code + 1, k + 1
                    code <<= 1
                tables[seg[q]], q = table, k
        elif marker == 0xC0:
            h, w, nc = struct.unpack(">HHB", seg[1:6])
            comps = [(seg[7 + 3 * i] >> 4, seg[7 + 3 * i] & 15) if nc > 1 else (1, 1) for i in range(nc)]
        elif marker == 0xDD:
            restart = struct.unpack(">H", seg)[0]
        p += 2 + n
        if marker == 0xDA:
            sel = [seg[2 + 2 * i] for i in range(len(comps))]
            break
    hm, vm = max(c[0] for c in comps), max(c[1] for c in comps)
    left = -(-w // (8 * hm)) * -(-h // (8 * vm))
    intervals = data[p:-2].replace(b"\xff\x00", b"\xff\xfe")  # (FE: no marker)
    cuts = [k for k in range(len(intervals) - 1) if intervals[k] == 0xFF and 0xD0 <= intervals[k + 1] <= 0xD7]
    parts = [intervals[a:b].replace(b"\xff\xfe", b"\xff")
             for a, b in zip([0] + [c + 2 for c in cuts], cuts + [len(intervals)])]
    out, phases = data[:p], [c for c, (sx, sy) in enumerate(comps) for _ in range(sx * sy)]
    for i, part in enumerate(parts):
        bits, pos = np.unpackbits(np.frombuffer(part, np.uint8)).tolist(), 0

        def symbol(table, pos):
            code = 0
            for length in range(1, 17):
                code = 2 * code + bits[pos + length - 1]
                if (length, code) in table:
                    return table[length, code], pos + length
            raise ValueError

        for _ in range(min(restart, left)):
            for c in phases:
                size, pos = symbol(tables[sel[c] >> 4], pos)
                pos, k = pos + size, 0
                while k < 63:
                    s, pos = symbol(tables[16 | (sel[c] & 15)], pos)
                    if s == 0:
                        break
                    k, pos = k + (s >> 4) + 1, pos + (s & 15)
        left -= min(restart, left)
        n = len(bits) - pos
        assert 0 <= n < 8
        for j in range(n):
            bits[pos + j] = pad(i, n) >> (n - 1 - j) & 1
        if i:
            out += bytes([0xFF, 0xD0 + (i - 1) % 8])
        out += np.packbits(np.array(bits, np.uint8)).tobytes().replace(b"\xff", b"\xff\x00")
    return out + b"\xff\xd9"


@pytest.mark.parametrize("mode,optimize", [("gray", False), ("420", True), ("444", False), ("422", True)])
def test_padding_bits_do_not_matter(cj, oracle_mod, mode, optimize):
    good = W.small_case(77, 200, 150, mode, 80, 1, "texture", optimize).data
    assert repad(good, lambda i, n: 127) == good
    rng = np.random.default_rng(5)
    files = [repad(good, lambda i, n: 0), repad(good, lambda i, n: 1), repad(good, lambda i, n: 15)]
    files += [repad(good, lambda i, n: int(rng.integers(128))) for _ in range(3)]
    want = oracle_mod.decode(good).pixels
    for f in files:
        ref = oracle_mod.decode(f)
        assert ref.error == 0 and np.array_equal(ref.pixels, want)
    for bits in (0, 128, 256, 512, 1024, 4096):
        with cj.Reader(sub_bits=bits) as r:
            for f in files:
                r.open_bytes(f)
                assert np.array_equal(r.pixels(), want)
        with cj.Batch(sub_bits=bits) as b:
            imgs, errs = b.decode(files)
            assert not any(errs) and all(np.array_equal(im, want) for im in imgs)
