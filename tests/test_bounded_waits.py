"""What the GEMM kernels do when a bounded wait runs out cannot be run on a shared GPU without copies in flight being
abandoned on purpose, so the rules the code has to keep are checked on its source."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parent.parent / "csrc" / "kernels"


def _source(name):
    """The file without comments."""
    return re.sub(r"//[^\n]*", "", (KERNELS / name).read_text())


@pytest.mark.parametrize("name", ["gemm_kernel.cuh", "gemm2_kernel.cuh", "gemm_small.cu"])
def test_a_role_waits_as_a_whole_warp(name):
    """Lanes of a warp can get different answers from a wait that runs out, and tcgen05.ld, cluster barriers and
    full-mask shuffles are undefined for half a warp: a result that decides what a role does comes from
    mbar_wait_warp."""
    decides = re.findall(r"(?:if \(!?|=\s*)(mbar_wait\w*)\(", _source(name))
    assert decides and set(decides) == {"mbar_wait_warp"}
