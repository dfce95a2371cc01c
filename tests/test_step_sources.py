"""What the step kernels' sources must not do: the pair step and the tail
kernel are launched while a kernel that writes the atoms' records may still
run, so they read no record through the read-only path (ld.global.nc, __ldg),
which asks for memory that is constant for the kernel's whole life.  The
neighbour lists, written at builds only, may be read that way."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "liggghts-public_b200", "csrc")


@pytest.mark.parametrize("name", ["gb2_step.cuh", "gb2_device.cuh", "gb2_split.cu"])
def test_records_are_read_by_ordinary_loads(name):
    code = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    assert "ld.global.nc" not in code
    for arg in re.findall(r"__ldg\(&(\S+?)\[", code):
        assert arg in ("D.rev", "D.nbr", "idx"), arg
