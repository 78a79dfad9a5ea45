"""Shared-memory bounds of the z operators on the tensor cores (csrc/iw_layout.h): every value that
a fragment reads lies inside what the launch asks for, at every nzloc the kernels take."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "iwrepo_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "iw_layout.h"
int main() {
  for (int N = 3; N <= kTcMaxN; ++N)
    std::printf("%d %d %d %d %d\n", N, tc_nt(N), tc_ap(N), tc_nc(N), tc_op_doubles(N));
}
"""


def test_fragments_of_the_last_operator_stay_in_bounds(tmp_path):
    src, exe = tmp_path / "layout.cpp", tmp_path / "layout"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    rows = [tuple(map(int, r.split())) for r in subprocess.run([str(exe)], check=True, capture_output=True,
                                                             text=True).stdout.splitlines()]
    assert [r[0] for r in rows] == list(range(3, 41))
    for n, nt, ap, nc, doubles in rows:
        # operand rows 4 kt + t (kt while 4 kt < N, t < 4), result rows 8 i + g (i < NT, g < 8)
        reads = [(4 * kt + t) * ap + 8 * i + g for kt in range(2 * nt) if 4 * kt < n for t in range(4)
                 for i in range(nt) for g in range(8)]
        assert 8 * nt >= n and nc >= n and max(reads) < doubles, n
        # zeroed or copied columns never overlap the next one
        assert ap >= n, n
