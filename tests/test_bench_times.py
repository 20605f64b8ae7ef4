"""The bench line's two times of a step are reported apart: the kernel alone and the chain's period."""
import pytest

import bench


@pytest.mark.parametrize("alone,chain", [(0.095, 0.086), (0.080, 0.086)])
def test_each_time_under_its_own_name(alone, chain):
    t = bench.step_times(200 * alone, 200, 1000 * chain, 1000)
    assert t["kernel_ms_avg"] == pytest.approx(alone) and t["chain_ms_per_step"] == pytest.approx(chain)
