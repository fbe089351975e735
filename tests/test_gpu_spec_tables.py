"""The speculative decode's shared-memory tables (CJSpecTab) and how the
images of a batch share them: images with DHT contents of their own beside
images that share one set, grey beside colour, long codes and positions up to
63, at the subsequence sizes where the decode's ring refills, checkpoints and
joins fall differently.  Every image must equal the oracle's decode bit for
bit."""
import numpy as np
import pytest

from cudajpeg_b200 import workloads as W

pytestmark = pytest.mark.gpu


def files(kind):
    if kind == "own tables":  # more distinct tables in a group of 8 warps than staging slots
        return [W.small_case(300 + k, 40 + 8 * k, 56, ["420", "444", "gray", "422"][k % 4], 50 + 3 * k, 0, "texture",
                             optimize=True).data for k in range(14)]
    if kind == "shared and own":
        return [W.small_case(400 + k, 64 + 24 * k, 72, ["gray", "420", "422"][k % 3], 80, [0, 3][k % 2], "smooth",
                             optimize=k % 4 == 3).data for k in range(12)]
    if kind == "grey only":
        return [W.small_case(500 + k, 33 + 16 * k, 47, "gray", 90).data for k in range(5)]
    if kind == "long codes":  # noise at high quality: 16-bit codes, blocks that end on position 63
        return [W.small_case(600 + k, 128, 96, m, q, ri, "noise").data
                for k, (m, q, ri) in enumerate([("444", 99, 0), ("420", 98, 1), ("gray", 100, 0), ("422", 97, 5)])]
    if kind == "flat":  # blocks of a few bits: more blocks than symbols per round
        from PIL import Image
        import io
        out = []
        for k, (w, h) in enumerate([(16, 16), (640, 480), (1000, 24)]):
            buf = io.BytesIO()
            Image.fromarray(np.full((h, w, 3), 90 + k, np.uint8), "RGB").save(buf, "JPEG", quality=30, subsampling=2)
            out.append(buf.getvalue())
        return out
    raise ValueError(kind)


@pytest.mark.parametrize("sub_bits", [128, 512, 1056, 4096])
@pytest.mark.parametrize("kind", ["own tables", "shared and own", "grey only", "long codes", "flat"])
def test_batches_equal_the_oracle(cj, oracle_mod, kind, sub_bits):
    fs = files(kind)
    for hyp in (True, False):
        with cj.Batch(sub_bits=sub_bits) as b:
            b.set_hypotheses(hyp)
            imgs, errs = b.decode(fs)
            for k, f in enumerate(fs):
                ref = oracle_mod.decode(f)
                assert ref.error == 0 and errs[k] == 0
                assert np.array_equal(imgs[k], ref.pixels), (kind, sub_bits, hyp, k)


@pytest.mark.parametrize("sub_bits", [128, 1024])
def test_single_files_equal_the_oracle(cj, oracle_mod, sub_bits):
    for kind in ("own tables", "long codes", "flat"):
        for f in files(kind)[:4]:
            with cj.Reader(sub_bits=sub_bits) as r:
                r.open_bytes(f)
                assert np.array_equal(r.pixels(), oracle_mod.decode(f).pixels), kind
