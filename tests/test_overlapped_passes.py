"""Sources of the kernels that start while the one before them still runs.

Read-only loads (__ldg, ld.global.nc) are defined for data that nothing writes
while the kernel runs, and griddepcontrol.wait does not order them: the passes
read what their predecessor writes with ordinary loads.
"""
import os
import re

import pytest

from simp_b200 import build


@pytest.mark.parametrize("name", ["passes.cu", "pass_common.cuh", "tile.cuh", "walls.cuh"])
def test_no_read_only_loads(name):
    with open(os.path.join(build.CSRC, name)) as f:
        code = re.sub(r"//.*", "", f.read())
    assert not re.findall(r"__ldg|__ldcv?\b|ld\.global\.nc|ld\.global\.L1::no_allocate", code)
