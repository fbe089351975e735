"""Index arithmetic of the coefficient write-out (cj_core.h, the code the
kernel compiles) at sizes no test image reaches, built for the host."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run_host(tmp_path, body):
    src = tmp_path / "t.cpp"
    src.write_text('#include <stdio.h>\n#include "cudajpeg_b200/csrc/cj_core.h"\nint main() {\n' + body + "\nreturn 0;\n}\n")
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", ROOT, str(src), "-o", exe], check=True)
    return subprocess.run([exe], check=True, capture_output=True, text=True).stdout


def test_any_block_of_an_image_is_stored_at_its_place(tmp_path):
    """A unit's blocks lie up to an image (2^28 blocks) from the warp's first unit, on either side."""
    out = run_host(tmp_path, """
      const long long at[] = {0, 1, (1 << 26) - 1, 1 << 26, (1 << 26) + 5, 201 * 1000 * 1000, 0x7FFFFFFF};
      for (long long b : at)
        for (int s = -1; s <= 1; s += 2)
          for (unsigned lane = 0; lane < 32; lane++) {
            const CJDone d = cj_done((int32_t)(s * b), lane);
            if (cj_done_chunk(d) != 8 * s * b || d.lane != lane) printf("%lld %u\\n", s * b, lane);
          }
      printf("done\\n");""")
    assert out == "done\n"


def test_positions_in_a_truncated_scans_padding_do_not_wrap(tmp_path):
    """2^34 bits of padding: the position stays behind the data, keeps its place in the window's ring of 8
    words, and its chunk index keeps up with it."""
    out = run_host(tmp_path, """
      const uint32_t data_end = 8u * CJ_MAX_SCAN_BYTES;
      uint32_t pos = data_end, cb = pos >> 7;
      uint64_t full = pos;
      for (uint32_t k = 0; full < 1ull << 34; k++) {
        const uint32_t step = 3 * (k % 32);  // a round of three symbols
        pos += step;
        full += step;
        cb = pos >> 7;
        cj_fold_position(pos, cb);
        if (pos < data_end || (pos & 255) != (full & 255) || cb != pos >> 7) {
          printf("%u %llu\\n", pos, (unsigned long long)full);
          break;
        }
      }
      printf("done\\n");""")
    assert out == "done\n"
