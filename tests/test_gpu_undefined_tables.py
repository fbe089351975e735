"""A file that uses a quantisation table it does not define decodes as with a
table of zeros, whatever was decoded before it and by whichever entry point."""
import numpy as np
import pytest

from cudajpeg_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_undefined_quantisation_table(cj):
    import ctypes as C

    import torch

    before = W.small_case(3, 80, 64, "gray", 60).data
    data = bytearray(W.small_case(4, 200, 40, "gray", 85).data)
    at = bytes(data).index(b"\xff\xdb")
    assert data[at + 4] == 0
    data[at + 4] = 1  # defines table 1, the scan uses table 0
    data = bytes(data)
    with cj.Reader() as r:
        r.open_bytes(data)
        want = r.pixels()
    assert (want == 128).all()
    for on_device in (True, False):
        with cj.Batch() as b:
            b.set_parse(on_device)
            imgs, errs = b.decode([before, data, before, data])
            assert not any(errs) and np.array_equal(imgs[1], want) and np.array_equal(imgs[3], want)
    out = torch.zeros(want.size, dtype=torch.uint8, device="cuda")
    w, h, c = C.c_int(), C.c_int(), C.c_int()
    for f, expect in ((before, None), (data, want), (before, None), (data, want)):
        err = cj.load().cjDecodeNoAlloc(f, len(f), C.c_void_p(out.data_ptr()), out.numel(), C.byref(w), C.byref(h),
                                        C.byref(c), None)
        assert err == 0
        if expect is not None:
            assert np.array_equal(out.cpu().numpy().reshape(expect.shape), expect)
