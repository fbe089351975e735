"""Progressive scans that follow one another inside one launch, against the
oracle: refinements block by block behind their predecessors (one interval per
scan), whole scans behind whole scans (restart intervals, few enough for all
to run at once), and a launch per level (more intervals than fit)."""
import io

import numpy as np
import pytest
from PIL import Image

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,q,sub,ri", [(48, 40, 90, 2, 0), (700, 513, 90, 2, 0), (515, 260, 95, 0, 0),
                                          (512, 384, 85, 2, 200), (384, 256, 92, 0, 300), (512, 512, 80, 2, 16)])
def test_scans_that_follow_one_another(cj, oracle_mod, w, h, q, sub, ri):
    rng = np.random.default_rng(w * h + ri)
    yy, xx = np.mgrid[0:h, 0:w]
    a = np.stack([128 + 70 * np.sin(xx / (7 + c)) * np.cos(yy / 11) + rng.normal(0, 14, (h, w)) for c in range(3)], -1)
    kw = {"restart_marker_blocks": ri} if ri else {}
    buf = io.BytesIO()
    Image.fromarray(np.clip(a, 0, 255).astype(np.uint8)).save(buf, "JPEG", quality=q, subsampling=sub, progressive=True,
                                                              **kw)
    data = buf.getvalue()
    ref = oracle_mod.decode(data)
    assert ref.error == 0
    with cj.Reader() as r:
        for _ in range(3):
            r.open_bytes(data)
            assert np.array_equal(r.pixels(), ref.pixels)
