"""The segments of the compact scheme's flux pass: a shape that was asked for is the one that
runs, the library's own fills the SMs (host build of gbh_cr_plan.h)."""
import os
import subprocess

from hypar_gb300 import build as B

SRC = r"""
#include <cstdio>
#include "gbh_cr_plan.h"
int main() {
  const int asked[] = {1, 3, 7, 32, 64, 4096};
  for (int a : asked) std::printf("%d ", gbh::cr_segment(a, 37, 37, 152));
  std::printf("%d %d %d %d\n", gbh::cr_segment(0, 37, 37, 152), gbh::cr_segment(0, 64, 4096, 152),
              gbh::cr_segment(0, 256, 65536, 152), gbh::cr_segment(0, 64, 4096, 76));
  return 0;
}
"""


def test_segments(tmp_path):
    src, exe = tmp_path / "plan.cpp", str(tmp_path / "plan")
    src.write_text(SRC)
    subprocess.check_call(["g++", "-std=c++17", "-I", B.CSRC, "-o", exe, str(src)])
    got = [int(v) for v in subprocess.check_output([exe], text=True).split()]
    assert got == [1, 3, 7, 32, 64, 4096, 2, 3, 32, 6]
    assert os.path.exists(os.path.join(B.CSRC, "gbh_cr_plan.h"))
