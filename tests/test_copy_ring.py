"""Where the digit GEMM's producer stops (csrc/copy_ring.h): the copies that may still be in flight, for every stage and tile
at which it can give up, against a record of what was issued.  Compiled for the host; no device."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ad_afqmc_prototype_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "copy_ring.h"
// Stages of `tiles` A tiles, issued one by one, then as many B tiles together; the producer stops after `issued` A tiles
// of stage `stages`.  last[p][j]: the last stage whose tile j went to buffer p.
int main() {
    const int tiles = 7;
    for (unsigned stages = 0; stages < 9; ++stages)
        for (int extra = 0; extra <= tiles; ++extra) {
            int a[2][tiles], b[2][tiles];
            for (int p = 0; p < 2; ++p)
                for (int j = 0; j < tiles; ++j) a[p][j] = b[p][j] = -1;
            for (unsigned v = 0; v < stages; ++v)
                for (int j = 0; j < tiles; ++j) a[v & 1][j] = b[v & 1][j] = (int)v;
            for (int j = 0; j < extra; ++j) a[stages & 1][j] = (int)stages;
            for (int p = 0; p < 2; ++p)
                for (int j = 0; j < tiles; ++j)
                    if (afq::ring_last(stages, extra, j, p) != a[p][j] || afq::ring_last(stages, 0, j, p) != b[p][j]) {
                        std::printf("stages %u extra %d tile %d buffer %d\n", stages, extra, j, p);
                        return 1;
                    }
        }
    return 0;
}
"""


def test_every_copy_in_flight_is_waited_for(tmp_path):
    src = tmp_path / "ring.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "ring"
    built = subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)],
                           capture_output=True, text=True)
    if built.returncode != 0 and "No such file" in built.stderr and "copy_ring.h" not in built.stderr:
        pytest.skip("no host compiler")
    assert built.returncode == 0, built.stderr
    ran = subprocess.run([str(exe)], capture_output=True, text=True)
    assert ran.returncode == 0, ran.stdout
