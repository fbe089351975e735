"""MCU-phase hypotheses at subsequence sizes that were set, up to and past the
hypothesis warps per SM at which they stop: every decode equals the oracle's,
with them and without."""
import numpy as np
import pytest

from cudajpeg_b200 import workloads as W

pytestmark = pytest.mark.gpu


# (warps of hypothesis decodes per SM of 148: about 14, 23, 29, 47)
@pytest.mark.parametrize("w,h,bits", [(1600, 1200, 256), (2048, 1536, 256), (1600, 1200, 128), (2048, 1536, 128)])
def test_reader_at_a_set_size(cj, oracle_mod, w, h, bits):
    data = W.small_case(w + bits, w, h, "420", 85, 0, "smooth").data
    with cj.Reader(sub_bits=bits) as r:
        r.open_bytes(data)
        assert np.array_equal(r.pixels(), oracle_mod.decode(data).pixels)


@pytest.mark.parametrize("n,bits", [(8, 1024), (8, 512), (8, 256)])  # about 9, 18 and 37
def test_batch_at_a_set_size(cj, oracle_mod, n, bits):
    files = [W.small_case(k, 1024, 768, "420", 80, 0, "smooth").data for k in range(n)]
    want = [oracle_mod.decode(f).pixels for f in files]
    for on in (True, False):
        with cj.Batch(sub_bits=bits) as b:
            b.set_hypotheses(on)
            imgs, errs = b.decode(files)
            assert not any(errs) and all(np.array_equal(x, y) for x, y in zip(imgs, want))
