"""Constants of the small DFTs, against 80-bit values."""

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "gpe_simulator_b200" / "csrc"
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

SOURCE = """
#include "gpe_fft.cuh"
#include <cstdio>
template <int R, int E = 1> void show() {
  constexpr gpe::CxCS w = gpe::cx_root(E, R);
  printf("%d %d %a %a\\n", R, E, w.c, w.s);
  if constexpr (E + 1 < R) show<R, E + 1>();
}
int main() { show<3>(); show<5>(); show<6>(); show<7>(); show<9>(); show<10>(); show<11>(); show<12>(); show<13>();
             show<14>(); show<15>(); }
"""


@pytest.mark.skipif(not Path(NVCC).exists(), reason="needs nvcc")
def test_roots_are_correctly_rounded(tmp_path):
    src, exe = tmp_path / "roots.cu", tmp_path / "roots"
    src.write_text(SOURCE)
    subprocess.run([NVCC, "-std=c++17", "--expt-relaxed-constexpr", "-I", str(CSRC), "-o", str(exe), str(src)], check=True)
    pi = np.longdouble("3.14159265358979323846264338327950288")
    seen = 0
    for line in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.splitlines():
        r, e, c, s = line.split()
        a = 2 * pi * np.longdouble(int(e)) / np.longdouble(int(r))
        for got, want in ((c, np.cos(a)), (s, np.sin(a))):
            got = float.fromhex(got)
            assert got == float(want) or (abs(want) < 1e-18 and got == 0.0), (r, e, got, want)
            seen += 1
    assert seen == 2 * sum(r - 1 for r in (3, 5, 6, 7, 9, 10, 11, 12, 13, 14, 15))
