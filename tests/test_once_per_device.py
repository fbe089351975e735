"""Set-up that belongs to a device (cj_once.h): made on every device, once, also
when several threads come first, and tried again where it failed."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

BODY = r"""
#include <stdio.h>
#include <thread>
#include <vector>
#include "cudajpeg_b200/csrc/cj_once.h"
static CJOncePerDevice attrs;
static std::atomic<int> calls[70];
static int answer[70];
static int make(int d) {
  return attrs.run(d, [=] { calls[d]++; return answer[d]; });
}
int main() {
  make(0), make(0), make(1), make(1), make(63);  // a second device has its own
  printf("%d %d %d %d\n", (int)calls[0], (int)calls[1], (int)calls[2], (int)calls[63]);
  answer[2] = 7;
  const int failed = make(2);
  answer[2] = 0;
  const int then = make(2);
  make(2);
  printf("%d %d %d\n", failed, then, (int)calls[2]);
  make(64), make(64);
  printf("%d\n", (int)calls[64]);
  std::vector<std::thread> t;
  for (int k = 0; k < 8; k++) t.emplace_back([] { for (int i = 0; i < 1000; i++) for (int d = 3; d < 20; d++) make(d); });
  for (auto& x : t) x.join();
  bool few = true;
  for (int d = 3; d < 20; d++) few = few && calls[d] >= 1 && calls[d] <= 8;
  printf("%d\n", few);
}
"""


def test_once_per_device(tmp_path):
    src, exe = tmp_path / "t.cpp", str(tmp_path / "t")
    src.write_text(BODY)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", ROOT, str(src), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split("\n")
    assert out[0] == "1 1 0 1"
    assert out[1] == "7 0 2"
    assert out[2] == "2"
    assert out[3] == "1"


def test_no_attribute_is_set_behind_a_process_wide_flag():
    """Every cudaFuncSetAttribute of the library runs per device: through CJOncePerDevice, an array by device,
    or on each call -- never behind one static flag for the process."""
    csrc = os.path.join(ROOT, "cudajpeg_b200", "csrc")
    for name in sorted(os.listdir(csrc)):
        if name.endswith((".cu", ".cuh")):
            text = open(os.path.join(csrc, name)).read()
            for at in [k for k in range(len(text)) if text.startswith("cudaFuncSetAttribute", k)]:
                before = text[max(0, at - 400):at]
                assert "static bool attr_set" not in before and "static bool attrs" not in before, name
