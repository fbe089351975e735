"""Batches whose files have Huffman tables of their own, by the number of files:
one warp of the entropy decode per group (few files) up to eight with eight
table sets, of which two are in shared memory and the others read from global
memory; alone and among files that share a set.  Every image must equal the
oracle's decode."""
import numpy as np
import pytest

from cudajpeg_b200 import workloads as W

pytestmark = pytest.mark.gpu


def distinct(shared):
    """13 files of a few blocks to a few hundred, noise among them (long codes)."""
    return [W.small_case(900 + k, 16 + 8 * (k % 6), 17 + 5 * (k % 9), ["420", "gray", "444", "422"][k % 4], 60 + 3 * k,
                         [0, 2][k % 3 == 1], ["texture", "noise", "smooth"][k % 3],
                         optimize=not (shared and k % 3)).data for k in range(13)]


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("n", [3, 60, 650, 1300, 2600])
@pytest.mark.parametrize("sub_bits", [0, 128])
def test_own_tables_by_batch_size(cj, oracle_mod, n, sub_bits, shared):
    files = distinct(shared)
    want = [oracle_mod.decode(f).pixels for f in files]
    with cj.Batch(sub_bits=sub_bits) as b:
        imgs, errs = b.decode([files[k % 13] for k in range(n)])
        assert not any(errs)
        for k in range(n):
            assert np.array_equal(imgs[k], want[k % 13]), k
