"""bench.py's roofline figures where a launch advances several iterations."""
import pytest

import bench


# 100 iterations one a launch; in 25 launches of four, which move a quarter
@pytest.mark.parametrize("launches,bpl,gbs", [(100, 240.0, 240.0), (25, 60.0, 60.0)])
def test_a_launch_moves_the_state_once(launches, bpl, gbs):
    got = bench.hbm_of(2, "f64", 10 ** 6, launches, 100, 100.0)
    assert got == (bpl, 100.0 / launches, pytest.approx(gbs))


def test_kernel_names():
    class Cav:
        kernel, dim = "march", 2
    assert bench.step_kernels(Cav, 100, 100) == "k_march2d"
    assert "k_march2d_levels" in bench.step_kernels(Cav, 25, 100)
    Cav.kernel, Cav.dim = "direct", 3
    assert bench.step_kernels(Cav, 100, 100) == "k_step3d"
