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


def test_epilogue_warps_that_meet_at_barriers_leave_together():
    """Barriers of the four epilogue warps have no limit, so none may depend on an answer that one warp got alone: the
    wait for a finished tile is agreed on where the epilogue has such barriers, and the abort flag is combined in the
    barrier instead of being read behind it."""
    fused = _source("gemm_fused.cu")
    for name in ("gemm_kernel.cuh", "gemm2_kernel.cuh"):
        assert len(re.findall(r"accumulator_wait<Epilogue>\(smem_u32\(&ctl->tmem_full", _source(name))) == 1
    for struct in re.findall(r"struct (\w+Epilogue) \{(.*?)\n\};", fused, re.S):
        meets = "epilogue_warps_" in struct[1]
        assert f"kWarpsMeet = {'true' if meets else 'false'};" in struct[1], struct[0]
    assert not re.findall(r"epilogue_warps_sync\(\);\s*if \(\*abort_flag", fused)
