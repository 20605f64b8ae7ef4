"""The marches' stage waits give one verdict per warp. Lanes poll an mbarrier and the clock apart; a
stage that lands around the limit would let some lanes of a warp leave while the others reach
warp-wide instructions (tensor-memory accesses, __syncwarp) without them."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flowcontrast_b200", "csrc")


@pytest.mark.parametrize("source", ["step2_kernel.cuh", "stepcol_kernel.cuh"])
def test_march_decides_by_warp(source):
    """arrive_wait returns on the warp's vote; a lane polls for itself only inside lane 0's branch."""
    text = open(os.path.join(CSRC, source)).read()
    body = re.search(r"auto arrive_wait = .*?\n  \};\n", text, re.S).group(0)
    decision, rest = body.split("return true;")
    assert "mbar_wait_warp(" in decision and "mbar_wait_bounded(" not in decision
    assert rest.index("if (lane == 0)") < rest.index("mbar_wait_bounded(") < rest.index("__syncwarp();")
    assert text.count("mbar_wait_bounded(") == body.count("mbar_wait_bounded(")


@pytest.mark.gpu
def test_lanes_at_the_limit_agree(built, ctx):
    alone, warp = ctx.selftest_warp_wait(limit_ms=160.0)
    assert alone == 0xAAAAAAAA             # the odd lanes, whose limit is later, saw the phase
    assert warp == 0
    with pytest.raises(built.FslbmError):
        built._check(built.lib().fslbm_selftest_warp_wait(ctx.handle, -1.0, None))
