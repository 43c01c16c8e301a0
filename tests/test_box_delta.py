"""Differences of box fractions (csrc/fpconv.h) over the whole range, compiled with checks for
signed overflow."""
import os
import subprocess

from conftest import ROOT

SRC = r'''
#include <cstdio>
#include <cstdint>
#include "fpconv.h"
int main() {
  const int64_t edge[9] = {-2147483648LL, -2147483647LL, -1500000000LL, -1, 0, 1, 1500000000LL, 2147483646LL, 2147483647LL};
  for (int64_t a : edge)
    for (int64_t b : edge) {
      int64_t d = (a - b) % 4294967296LL;
      d += d < -2147483648LL ? 4294967296LL : d > 2147483647LL ? -4294967296LL : 0;
      if (emdee::box_delta((int)a, (int)b) != d) return 1;
    }
  std::puts("ok");
}
'''


def test_wraps(tmp_path):
    (tmp_path / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fsanitize=signed-integer-overflow", "-fno-sanitize-recover=all", "-I",
                    os.path.join(ROOT, "emdee_gb300", "csrc"), str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    assert subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, check=True).stdout == "ok\n"
