"""Rules of the kernel sources that no run can show."""
import os

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "openmxp_b200", "csrc")


@pytest.mark.parametrize("name", ["batched.cu", "diag_coop.cu", "dense_tile.cuh"])
def test_no_read_only_loads_of_what_the_kernel_writes(name):
    """ld.global.nc is defined only for data that nothing writes while the kernel runs;
    these kernels read back factors that they wrote themselves."""
    text = open(os.path.join(CSRC, name)).read()
    assert "__ldg(" not in text and "ld.global.nc" not in text
