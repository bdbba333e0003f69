"""Which page-locked arrays a kernel may read itself: those that one locked range
holds whole (ela3d_hostrange.h, compiled for the host)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROG = r"""
#include <stdio.h>
#include "ela3d_hostrange.h"
int main() {
  unsigned long long s, n, p, b;
  while (scanf("%llu %llu %llu %llu", &s, &n, &p, &b) == 4) printf("%d\n", (int)ela3d::range_holds(s, n, p, b));
}
"""


def test_range_holds_an_array_whole_or_not_at_all(tmp_path):
    src, exe = tmp_path / "r.cpp", tmp_path / "r"
    src.write_text(PROG)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "ela3d_gb300", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    top = (1 << 64) - 1
    rows = [(s, n, p, b) for s in (0, 4096, 1 << 40) for n in (1, 4095, 4096, 8192)
            for p in (0, s - 1, s, s + 1, s + n - 1, s + n, s + n + 1) for b in (0, 1, n - 1, n, n + 1, 1 << 30) if p >= 0 <= b]
    rows += [(top - 4095, 4095, top - 4095, 4095), (top - 4095, 4095, top - 4095, 4096), (top - 100, 100, top - 50, top),
             (0, top, 1, top - 1), (0, top, 1, top)]
    out = subprocess.run([str(exe)], input="\n".join("%d %d %d %d" % r for r in rows), capture_output=True, text=True,
                         check=True).stdout.split()
    want = [str(int(b > 0 and s <= p and p + b <= s + n)) for s, n, p, b in rows]
    assert out == want and "0" in want and "1" in want
