"""Progressive scans longer than the chunks their decode works in (2048 blocks
of a first scan, 256 of a refinement scan, 16384 bits), end-of-band runs across
chunks, scans that end in the middle of one, and intervals of a few bits.  Every
image must equal the oracle's decode (ITU T.81 Annex G) bit for bit."""
import io

import numpy as np
import pytest
from PIL import Image

pytestmark = pytest.mark.gpu


def content(kind, w, h, seed):
    rng = np.random.default_rng(seed)
    a = np.full((h, w, 3), 120, np.uint8)
    if kind == "noise":
        a = rng.integers(0, 256, (h, w, 3)).astype(np.uint8)
    elif kind == "islands":  # runs of empty blocks longer than a chunk, detail between them
        for _ in range(6):
            y, x = int(rng.integers(0, max(1, h - 12))), int(rng.integers(0, max(1, w - 12)))
            a[y:y + 12, x:x + 12] = rng.integers(0, 256, a[y:y + 12, x:x + 12].shape)
    elif kind == "smooth":
        yy, xx = np.mgrid[0:h, 0:w]
        for c in range(3):
            a[..., c] = np.clip(128 + 80 * np.sin(xx / (9 + c)) * np.cos(yy / 13) + rng.normal(0, 6, (h, w)), 0, 255)
    return a


CASES = [(k, w, h, q, sub, ri) for k, w, h, q, sub, ri in [
    ("islands", 640, 512, 90, 2, 0), ("islands", 1030, 130, 75, 0, 0), ("flat", 512, 512, 80, 2, 0),
    ("noise", 130, 128, 97, 0, 0), ("noise", 400, 300, 50, 2, 0), ("smooth", 512, 1040, 92, 1, 0),
    ("smooth", 384, 352, 85, 2, 1), ("noise", 96, 90, 99, 1, 7), ("islands", 256, 256, 60, 2, 40)]]


@pytest.mark.parametrize("kind,w,h,q,sub,ri", CASES)
@pytest.mark.parametrize("grey", [False, True])
def test_chunked_scans_equal_the_oracle(cj, oracle_mod, kind, w, h, q, sub, ri, grey):
    a = content(kind, w, h, w + h + q)
    img = Image.fromarray(a[..., 0], "L") if grey else Image.fromarray(a, "RGB")
    kw = {} if grey else {"subsampling": sub}
    if ri:
        kw["restart_marker_blocks"] = ri
    buf = io.BytesIO()
    img.save(buf, "JPEG", quality=q, progressive=True, **kw)
    data = buf.getvalue()
    ref = oracle_mod.decode(data)
    assert ref.error == 0
    with cj.Reader() as r:
        for _ in range(2):
            r.open_bytes(data)
            assert np.array_equal(r.pixels(), ref.pixels)
