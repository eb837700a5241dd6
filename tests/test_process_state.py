"""The library's entry points may be called for several devices and from
several threads, each with its own context: a kernel's attributes belong to a
device, so no function remembers in a static flag or counter that it has done
something once in this process. Read from the sources: the effect on a second
device cannot be seen on a machine with one."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "grasp_gb300", "csrc")
FLAG = re.compile(r"^\s+static\s+(?:volatile\s+)?(?:bool|int|unsigned|long|size_t|u?int\d+_t)\b[^;(]*[;=]", re.M)


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.c*"))), ids=os.path.basename)
def test_no_static_flags_in_functions(path):
    assert not FLAG.findall(open(path).read())
