"""The step kernel's instantiations keep their loops in registers: spilled
bytes as the assembler reports them at the build. Resident stepping with 184
bytes of spill loads a thread took 10% longer a call than with none."""

import os
import re

import pytest

import nemo_b200.build as b


def _spills():
    b.build()
    with open(os.path.join(b.BUILD, "kernels.cu.o.ptxas")) as f:
        text = f.read()
    found = {}
    for m in re.finditer(r"k_cyclesILb([01])ELj(\d+)ELi([012])ELb([01])E.*?(\d+) bytes spill stores, (\d+) bytes spill loads",
                         text, re.S):
        smem, threads, mode, hh, stores, loads = map(int, m.groups())
        found[smem, threads, mode, hh] = stores + loads
    return found


# mode 0: several cycles a launch, 1: one step, 2: resident stepping
@pytest.mark.parametrize("mode,most", [(0, 0), (1, 96), (2, 0)])
def test_spills(mode, most):
    spills = _spills()
    assert len(spills) == 36
    for smem in (0, 1):
        assert spills[smem, 1024, mode, 0] <= most, smem
