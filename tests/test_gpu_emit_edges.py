"""Output rows of any alignment, against the oracle, byte for byte.

RGB, planar, NV12 and fancy-upsampled output is written in groups that start
at aligned addresses, with single bytes at a row's ends; the groups shift with
the width and the row.  Every width residue mod 16, widths around a 256-pixel
strip and below one group, and odd heights, for each chroma form.
"""
import numpy as np
import pytest

from cudajpeg_b200 import workloads as W

pytestmark = pytest.mark.gpu

WIDTHS = [1, 2, 3, 5, 7] + list(range(33, 49)) + [255, 256, 257, 258, 511, 515]


@pytest.mark.parametrize("mode", ["420", "422", "444", "gray"])
def test_rows_of_any_alignment(cj, oracle_mod, mode):
    files = [W.small_case(700 + k, w, 9 + k % 13, mode, 80, 0, "noise").data for k, w in enumerate(WIDTHS)]
    refs = [oracle_mod.decode(f, fancy=True) for f in files]
    got = {}
    for fmt in (cj.OUTPUT_RGB, cj.OUTPUT_PLANAR, cj.OUTPUT_NV12, cj.OUTPUT_RGB_FANCY):
        with cj.Batch() as b:
            b.set_output(fmt, cj.IDCT_INT)
            got[fmt], errs = b.decode(files)
        assert list(errs) == [r.error for r in refs]
    assert sum(r.error == 0 for r in refs) >= len(WIDTHS) - 5  # (tiny images the format limits refuse)
    for k, (w, r) in enumerate(zip(WIDTHS, refs)):
        if r.error:
            continue
        planes = [p[: c.height, : c.width] for p, c in zip(r.planes, r.comps)]
        assert np.array_equal(got[cj.OUTPUT_RGB][k], r.pixels), w
        if r.nch == 1:
            for fmt in got:
                assert np.array_equal(got[fmt][k], r.pixels), (w, fmt)
            continue
        assert np.array_equal(got[cj.OUTPUT_RGB_FANCY][k], r.fancy_rgb), w
        for c in range(3):
            assert np.array_equal(got[cj.OUTPUT_PLANAR][k][c], planes[c]), (w, c)
        y, uv = got[cj.OUTPUT_NV12][k]
        assert np.array_equal(y, planes[0]), w
        assert np.array_equal(uv[..., 0], planes[1]) and np.array_equal(uv[..., 1], planes[2]), w
