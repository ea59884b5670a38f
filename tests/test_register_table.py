"""The mixed Taylor kernel's split (csrc/k_mixed.cu) counts how many CTAs an SM holds from a table of registers by rows a
thread: the table against what the compiler takes, rounded up to its allocation of eight.  No device."""
import os
import re
import shutil
import subprocess

import pytest

from ad_afqmc_prototype_gb300 import build

SOURCE = os.path.join(build.CSRC, "k_mixed.cu")


def test_table_is_what_the_compiler_takes(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    with open(SOURCE) as f:
        table = [int(v) for v in re.search(r"regs\[9\] = \{([^}]*)\}", f.read()).group(1).split(",")]
    r = subprocess.run([nvcc, *build.ARCH, *build.NVFLAGS, "-Xptxas", "-v", "-c", SOURCE, "-o", str(tmp_path / "k.o")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    used = {}
    for rows, n in re.findall(r"Compiling entry function '\w*k_trotter_mixedILi(\d)ELi\d+E.*?Used (\d+) registers",
                              r.stderr + r.stdout, re.S):
        used[int(rows)] = max(used.get(int(rows), 0), (int(n) + 7) // 8 * 8)
    assert used == {rows: table[rows] for rows in range(1, 9)}
