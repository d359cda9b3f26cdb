"""The batch autotuner times what a run launches."""
import pytest

pytestmark = pytest.mark.gpu


def test_tuner_times_the_launches_a_run_is_made_of(pkg):
    # launches of four steps, whatever number of steps was asked for
    b = pkg.Batch(2, [dict(nx=128, ny=128)] * 4)
    b.initial()
    b.step(1)
    i0, l0 = b.members[0].itc, pkg.lib().lbm_kernel_launches()
    r = b.tune(steps=4)
    steps, launches = b.members[0].itc - i0, pkg.lib().lbm_kernel_launches() - l0
    assert r["mlups"] > 0 and launches * 3 <= steps, (steps, launches)
    b.close()
