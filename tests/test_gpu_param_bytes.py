"""The bytes a reader reports as copied to the device beside the file's own."""
import pytest

from cudajpeg_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_param_bytes_count_the_whole_block(cj):
    """Header, plan and control block go in one copy: four Huffman tables (16 counts and 256 symbols each), four
    16-bit quantisation tables and a counter per SM slot are in it, whatever the rest."""
    with cj.Reader() as r:
        r.open_bytes(W.small_case(1, 64, 48, "420").data)
        assert r.info()["param_bytes"] >= 4 * (16 + 256) + 4 * 64 * 2 + 256 * 4
