"""The row index of a probe block's element on the host: blocks below, at and
past 2^32 elements (a graph of that size does not fit a GPU's memory)."""
import os
import subprocess

from conftest import ROOT

MAIN = r"""
#include <cstdio>
#include <initializer_list>
#include "probe_rows.hpp"
int main() {
  const long B = 1L << 32;
  int bad = 0;
  for (int P = 1; P <= 16; P++)
    for (long len : {1000L * P, B - 1, B, B + 1, B + 16L * P, 16L * 0x7fffffffL})
      for (long t : {0L, 1L, (long)P, len / 2, B - 2, B - 1, B, B + 1, B + P, len - 1})
        if (t < len)
          bad += (tbsla_gpu::probe_rows_wide(len) ? tbsla_gpu::probe_row<true>(t, P) : tbsla_gpu::probe_row<false>(t, P)) != t / P;
  printf("%d\n", bad);
}
"""


def test_rows(tmp_path):
    (tmp_path / "m.cpp").write_text(MAIN)
    exe = str(tmp_path / "m")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "tbsla_gb300", "csrc"), str(tmp_path / "m.cpp"),
                    "-o", exe], check=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True).stdout.strip() == "0"
