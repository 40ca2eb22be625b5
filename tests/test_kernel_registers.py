"""Registers of the pass kernels that transform lengths of radices 2 to 5, from
the compiler's report of this build: stages of radix 7 and above, which take up
to 250, stay out of every kernel such lengths run (a register allocation covers
everything a kernel calls)."""
import os
import re

import pytest


def registers(M, unit):
    path = os.path.join(os.path.dirname(M.LIB_PATH), "..", "_build", unit + ".o.ptxas")
    text = open(path).read()
    return {m.group(1): int(m.group(2))
            for m in re.finditer(r"Compiling entry function '(\w+)'.*?Used (\d+) registers", text, re.S)}


# mangled: f float, d double; the last Lb is ODD (k_x_forward: 3 components).  The
# limits are 64K registers over the CTAs per SM that these kernels run at.
LIMITS = [("kernels_f32.cu", "k_x_forwardIfLi3ELb0E", 64), ("kernels_f32.cu", "k_x_inverseIfLb0E", 64),
          ("kernels_f32.cu", "k_col_passIfLb0ELb0E", 80), ("kernels_f32.cu", "k_col_passIfLb1ELb0E", 80),
          ("kernels_f32.cu", "k_rowsIfLb0E", 128), ("kernels_f32.cu", "k_rowsIfLb1E", 128),
          ("kernels_f64.cu", "k_x_forwardIdLi3ELb0E", 128), ("kernels_f64.cu", "k_x_inverseIdLb0E", 128),
          ("kernels_f64.cu", "k_col_passIdLb0ELb0E", 144), ("kernels_f64.cu", "k_rowsIdLb0E", 184)]


@pytest.mark.parametrize("unit,kernel,limit", LIMITS, ids=lambda v: str(v))
def test_registers_without_odd_stages(M, unit, kernel, limit):
    found = [n for name, n in registers(M, unit).items() if kernel in name]
    assert len(found) == 1 and found[0] <= limit
