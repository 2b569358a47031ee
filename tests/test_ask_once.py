"""csrc/ask_once.h: a query whose answer is kept. A failed query (the cluster occupancy on a device that could not answer just then) must not
be kept as an answer for the life of the process. Host code: compiled and run with the host compiler."""

import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tilefish_b200", "csrc")
PROGRAM = r"""
#include "ask_once.h"
int main() {
  std::atomic<int> slot{0};
  int asked = 0;
  auto fails = [&] { ++asked; return -1; };
  auto answers = [&] { ++asked; return 47; };
  if (tf::ask_once(slot, fails) != 0 || asked != 1) return 1;
  if (tf::ask_once(slot, answers) != 47 || asked != 2) return 2;  // asked again after a failure
  if (tf::ask_once(slot, fails) != 47 || asked != 2) return 3;    // kept from then on
  std::atomic<int> zero{0};
  auto none = [&] { ++asked; return 0; };
  if (tf::ask_once(zero, none) != 0 || tf::ask_once(zero, none) != 0 || asked != 3) return 4;  // 0 is an answer
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_a_failed_query_is_asked_again(tmp_path):
    (tmp_path / "main.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "main")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-o", exe, str(tmp_path / "main.cpp")], check=True)
    assert subprocess.run([exe]).returncode == 0
    assert "ask_once(cached[dev][splits]" in open(os.path.join(CSRC, "gemm_blockscaled.cu")).read()
