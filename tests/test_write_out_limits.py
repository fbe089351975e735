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
