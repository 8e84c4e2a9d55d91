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


@pytest.mark.parametrize("name", ["gemm_kernel.cuh", "gemm2_kernel.cuh", "gemm_small.cu"])
def test_a_producer_stays_until_its_loads_have_landed(name):
    """Shared memory must not go away under a load in flight, whichever role gave up first: the last thing the
    producer does, on every path, is to wait (bounded) for its last loads, without asking the abort flag."""
    text = _source(name)
    producer = text[re.search(r"if \(warp == 0\) \{\s*uint32_t", text).start():]
    producer = producer[:producer.index("} else if (warp == 1)")]
    assert re.search(r"loads_land\(&ctl->full\[0\], NS, [^;]*\);\s*(if \(!ok\) loads_land\([^;]*;\s*\})?\s*$", producer), producer[-300:]
    land = _source("gemm_kernel.cuh")
    land = land[land.index("void loads_land"):]
    land = land[:land.index("\n}")]
    assert "abort" not in land and "budget_ns) return;" in land


def test_a_communication_cta_that_gives_up_lets_its_loads_land():
    fused = _source("gemm_fused.cu")
    comm = fused[fused.index("bulk_load("):]
    assert re.search(r"if \(!ok\) \{\s*loads_land\(s_full, [^;]*n_loaded[^;]*;\s*return;", comm)
