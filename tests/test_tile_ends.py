"""Tiles whose end lies past the largest int are not taken for whole ones (CPU: the
predicate that the kernels' epilogues use, against the same in 64 bits)."""
import subprocess

from tests.conftest import ROOT

PROGRAM = r"""
#include <climits>
#include <cstdio>
#include "common.cuh"
int main() {
  const int T = 128;
  int wrong = 0;
  for (int ji : {MUBLIS_L3_ALL, MUBLIS_L3_LOWER, MUBLIS_L3_UPPER})
    for (int m : {1, 127, 128, 129, 256, 300, INT_MAX - 128, INT_MAX - 127, INT_MAX - 1, INT_MAX})
      for (int n : {1, 127, 128, 129, 256, 300, INT_MAX - 128, INT_MAX - 127, INT_MAX - 1, INT_MAX})
        for (int a = 0; a < 3; ++a)
          for (int b = 0; b < 3; ++b)
            for (int back = 0; back < 4; ++back) {
              const long last_m = (m - 1L) / T, last_n = (n - 1L) / T;
              const long tm = back & 1 ? last_m - a : a, tn = back & 2 ? last_n - b : b;
              if (tm < 0 || tn < 0 || tm > last_m || tn > last_n) continue;
              const long m0 = tm * T, n0 = tn * T;
              const bool want = m0 + T <= m && n0 + T <= n &&
                                (ji == MUBLIS_L3_ALL || (ji == MUBLIS_L3_LOWER ? n0 + T <= m0 : m0 + T <= n0));
              wrong += want != b200_whole_tile(m, n, (int)tm, (int)tn, T, ji);
            }
  printf("%d\n", wrong);
  return wrong != 0;
}
"""


def test_tiles_at_the_largest_sizes(tmp_path):
    src, exe = tmp_path / "tiles.cpp", tmp_path / "tiles"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-fsanitize=signed-integer-overflow", "-fno-sanitize-recover",
                    f"-I{ROOT / 'mublis_b200' / 'csrc'}", f"-I{ROOT / 'include'}",
                    "-I/usr/local/cuda/include", str(src), "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True, timeout=60)


def test_epilogues_use_it():
    """No epilogue adds up a tile's end in 32 bits."""
    for name in ("gemm_dmma.cu", "gemm_ffma.cu"):
        text = (ROOT / "mublis_b200" / "csrc" / name).read_text()
        assert "b200_whole_tile(p.m, p.n, tm, tn, BM, p.ji)" in text, name
        assert "(tm + 1) * BM" not in text and "(tn + 1) * BN" not in text, name
        assert "int i0 = tm * BM" not in text, name
