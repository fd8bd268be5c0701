"""The x1 march addresses a column by 32-bit byte offsets (csrc/xmarch.cuh: a
line's place `t.q`, the steps `qx` from x to x and `qc` from component to
component). `x_offsets_fit` (csrc/xmarch_plan.h) admits exactly the columns whose
last stored byte such offsets reach. No GPU needed."""
import ctypes as C
import os
import subprocess

import pytest

from conftest import ROOT

SRC = r"""
#include "xmarch_plan.h"
extern "C" int fits(int n1, int n2, int n3) { return eqd::x_offsets_fit(n1, n2, n3); }
extern "C" int row_length(int n2) { return eqd::x_row_length(n2); }
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("xplan")
    src, out = d / "p.cpp", d / "p.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "earthquakediffinitive.jl_b200", "csrc"), "-o", str(out), str(src)], check=True)
    return C.CDLL(str(out))


def offsets(plan, n1, n2, n3):
    """The last element's byte offset as the kernel forms it, and in full."""
    n2p = plan.row_length(n2)
    lead, m = 3, 2 ** 32
    i2, i3, x, comp = n2 - 1, n3 - 1, n1 - 1, 2
    q = 4 * (3 * n1 * n3 * n2p + i3 * n2p + i2 + lead)
    qx = 4 * n3 * n2p
    qc = qx * n1
    return (q % m + x * (qx % m) + comp * (qc % m)) % m, q + x * qx + comp * qc, 4 * 6 * n1 * n3 * n2p


@pytest.mark.parametrize("n1,n2,n3", [
    (9, 9, 9), (9, 17, 17), (21, 81, 81), (33, 129, 129), (21, 1601, 1601), (33, 2201, 2201), (21, 2900, 2900),
    (16, 3197, 3495), (16, 3197, 3496), (21, 3201, 3201), (33, 3301, 3301), (9, 9, 1 << 22), (9, 20000, 20000)])
def test_offsets_fit(plan, n1, n2, n3):
    wrapped, full, size = offsets(plan, n1, n2, n3)
    assert bool(plan.fits(n1, n2, n3)) == (size <= 2 ** 32)
    if plan.fits(n1, n2, n3):
        assert wrapped == full
