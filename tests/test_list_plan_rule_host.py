"""Which systems ask for a list build (``asks_build``, compiled for the host): a
running one whose flag is raised.  A system that finished outside its skin, one
admitted and not armed yet, and a slot evicted with a plan pending keep their
flag raised and must not have the list plan made in every step."""
import itertools
import os
import subprocess

import pytest

from gliding_collective_rotation_b200 import build as B

MAIN = r"""
#include <cstdio>
#include "gcr_device.cuh"
int main()
{
    int v[5];
    while (scanf("%d %d %d %d %d", v, v + 1, v + 2, v + 3, v + 4) == 5) {
        gcr::SysP p{};
        gcr::SysS s{};
        s.rebuild = v[0];
        s.active = v[1];
        s.flags = v[2];
        p.calc_wca = v[3];
        p.fixed = v[4];
        printf("%d\n", gcr::asks_build(p, s) ? 1 : 0);
    }
    return 0;
}
"""


def test_only_running_systems_ask(tmp_path):
    try:
        nvcc = B.nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    src, exe = tmp_path / "asks.cu", tmp_path / "asks"
    src.write_text(MAIN)
    subprocess.run([nvcc, *B.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", os.path.abspath(B.CSRC), "-o",
                    str(exe), str(src)], check=True)
    # flags: none, cell overflow, series full (not fatal), wait expired
    cases = list(itertools.product((0, 1), (0, 1), (0, 1, 32, 64), (0, 1), (0, 1)))
    out = subprocess.run([str(exe)], input="\n".join(" ".join(map(str, c)) for c in cases), capture_output=True,
                         text=True, check=True).stdout.split()
    assert [int(x) for x in out] == [int(r and a and f in (0, 32) and w and not fx) for r, a, f, w, fx in cases]
