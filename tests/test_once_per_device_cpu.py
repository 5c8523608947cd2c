"""Kernels' permissions are a device's own: they are asked for on every device, and again after a refusal."""
import re
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "uniserve_v1_b200" / "csrc"

PROGRAM = """
#include "include/us_once.h"
#include <cstdio>
#include <initializer_list>
int main() {
  us::OncePerDevice once;
  int asked[70] = {0}, refuse = 1;
  auto on = [&](int d) { return once(d, [&] { ++asked[d]; return d == 2 && refuse ? 7 : 0; }); };
  int rc = 0;
  for (int round = 0; round < 3; ++round) {
    for (int d : {0, 1, 2, 63, 69}) {
      const int got = on(d);
      if (got != (d == 2 && refuse ? 7 : 0)) rc = 1;
    }
    refuse = 0;
  }
  printf("%d %d %d %d %d\\n", asked[0], asked[1], asked[2], asked[63], asked[69]);
  return rc;
}
"""


def test_asked_once_for_every_device(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["1", "1", "2", "1", "3"]


@pytest.mark.parametrize("name", ["chunk_delta.cu", "vector_delta.cu"])
def test_no_permission_for_the_first_device_alone(name):
    text = (CSRC / name).read_text()
    assert "cudaFuncSetAttribute" not in text and not re.search(r"static (bool|int) ", text)
