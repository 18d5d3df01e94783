"""div_nr and rcp_fast, the kernels' branch-free division and reciprocal, against the operator.

div_nr ends with the residual correction, which leaves half a unit in the last place and a
term of 2^-22 of it: at most one unit off, and only for quotients that close to a tie, which
2^24 random ones meet a few times.  rcp_fast ends with a product whose factor is rounded to
2^-53: within 1.5 units of the reciprocal, so two of the rounded one."""
import ctypes as C
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_against_the_operator(tmp_path):
    so = str(tmp_path / "division_check.so")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared",
                    "-Xcompiler", "-fPIC", "-o", so, os.path.join(HERE, "division_check.cu")], check=True)
    out = (C.c_ulonglong * 6)()
    n = 1 << 24
    assert C.CDLL(so).division_check(out, C.c_int(n)) == 0
    worst, differ = out[::2], out[1::2]
    assert worst[0] <= 1 and worst[1] <= 1 and worst[2] <= 2, (worst, differ)
    assert differ[0] <= n // 10**4 and differ[1] <= n // 10**4, differ
