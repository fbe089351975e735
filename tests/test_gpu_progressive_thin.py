"""Progressive scans of many short restart intervals, decoded by a thread each,
alone and between scans decoded by a CTA per interval, against the oracle; and
such files with a damaged byte."""
import io

import numpy as np
import pytest
from PIL import Image

from cudajpeg_b200 import workloads as W

pytestmark = pytest.mark.gpu


def encode(w, h, q, sub, ri, grey=False):
    a = W.smooth_content(np.random.default_rng(w * 7 + h), w, h, 3)
    buf = io.BytesIO()
    kw = {} if grey else {"subsampling": sub}
    Image.fromarray(a[..., 0] if grey else a).save(buf, "JPEG", quality=q, progressive=True, restart_marker_blocks=ri, **kw)
    return buf.getvalue()


# (an interval per MCU: all scans by threads; 2 to 16 MCUs: some of a frame's; 64: none)
@pytest.mark.parametrize("w,h,q,sub,ri", [(512, 512, 60, 2, 1), (513, 511, 95, 2, 1), (1024, 768, 60, 2, 2), (1000, 700, 80, 1, 3),
                                          (640, 480, 90, 0, 1), (1024, 768, 60, 2, 12), (1024, 768, 60, 2, 16),
                                          (2048, 1536, 60, 2, 16), (1024, 768, 60, 2, 64), (300, 200, 75, 2, 1)])
@pytest.mark.parametrize("grey", [False, True])
def test_short_intervals(cj, oracle_mod, w, h, q, sub, ri, grey):
    data = encode(w, h, q, sub, ri, grey)
    ref = oracle_mod.decode(data)
    assert ref.error == 0
    with cj.Reader() as r:
        for _ in range(2):
            r.open_bytes(data)
            assert np.array_equal(r.pixels(), ref.pixels)


@pytest.mark.parametrize("ri", [1, 8])
def test_damaged_intervals(cj, oracle_mod, ri):
    good = encode(512, 384, 80, 2, ri)
    rng = np.random.default_rng(ri)
    outcomes = set()
    with cj.Reader() as r:
        for _ in range(24):
            bad = bytearray(good)
            at = int(rng.integers(len(bad) // 3, len(bad) - 2))
            while bad[at] == 0xFF or bad[at - 1] == 0xFF or bad[at + 1] == 0xFF:
                at -= 1
            bad[at] ^= int(rng.integers(1, 255))
            if bad[at] == 0xFF:
                bad[at] ^= 1
            ref = oracle_mod.decode(bytes(bad))
            err = r.open_bytes(bytes(bad), check=False)
            # (the oracle also refuses an interval that ends before its marker)
            assert err == 0 or ref.error != 0
            outcomes.add(ref.error == 0)
            if ref.error == 0:
                assert np.array_equal(r.pixels(), ref.pixels)
    assert outcomes == {True, False}
