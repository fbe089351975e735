"""A wait between thread blocks that runs out (a limit of one poll) ends a
reader's decode with an error, and the reader's next decode is right."""
import io

import numpy as np
import pytest
from PIL import Image

from cudajpeg_b200 import workloads as W

pytestmark = pytest.mark.gpu


def file(progressive):
    if not progressive:
        return W.small_case(11, 640, 480, "420", 80).data
    buf = io.BytesIO()
    Image.fromarray(W.smooth_content(np.random.default_rng(3), 512, 384, 3)).save(buf, "JPEG", quality=85,
                                                                                 progressive=True)
    return buf.getvalue()


@pytest.mark.parametrize("progressive", [False, True])
def test_a_wait_that_runs_out(cj, oracle_mod, progressive):
    data = file(progressive)
    want = oracle_mod.decode(data).pixels
    with cj.Reader() as r:
        for _ in range(3):
            r.set_wait_limit(1)
            assert r.open_bytes(data, check=False) == cj.CUDA_KERNEL_LAUNCH_ERROR
            r.set_wait_limit(0)
            r.open_bytes(data)
            assert np.array_equal(r.pixels(), want)
