"""The fast build's 3D march on the GPU: against the direct-load kernel at ragged
sizes (the shortest axes, tiles of one row of remainder fewer than a tile, both
tile heights, both directions of the walk), and in slabs, whose segments start
and end elsewhere.

Tolerance against the direct-load kernel: both form every interpolated value by
the same operations and differ at most in how the compiler contracts the
collision, a few units in the last place of O(1) populations per step (32
operations of half a unit each); 12 steps at most add up: 12 x 16 units."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cavity(pkg, shape, storage, kernel, steps, tiley=0):
    nx, ny, nz = shape
    m = pkg.lbm.mesh_box(nx, ny, nz, 1.0, ny / nx, nz / nx, "tanh", 1.5)
    c = pkg.Cavity(3, nx, ny, nz, Ra=1e5, Pr=0.71, coords=m, storage=storage, kernel=kernel)
    if tiley:
        c.set_option(pkg.lbm.OPT_TILEY, tiley)
    c.initial()
    c.step(steps)
    return c


@pytest.mark.parametrize("storage", ["f64", "f32"])
@pytest.mark.parametrize("shape,tiley", [((33, 18, 3), 4), ((40, 10, 4), 4), ((20, 16, 5), 8), ((64, 27, 6), 4),
                                         ((65, 12, 40), 8), ((35, 31, 29), 4)])
@pytest.mark.parametrize("steps", [1, 2, 11])
def test_march_matches_the_direct_kernel(pkg, shape, tiley, storage, steps):
    a = cavity(pkg, shape, storage, "direct", steps)
    b = cavity(pkg, shape, storage, "march", steps, tiley)
    assert (a.kernel, b.kernel) == ("direct", "march")
    unit = 2.0 ** -52 if storage == "f64" else 2.0 ** -23
    for k, v in a.macro().items():
        assert np.abs(b.macro()[k] - v).max() <= 12 * 16 * unit, k
    a.close()
    b.close()


@pytest.mark.parametrize("nslabs", [2, 3])
@pytest.mark.parametrize("storage", ["f64", "f32"])
def test_slabs_of_the_fast_build_are_bitwise(pkg, storage, nslabs):
    nx, ny, nz = 40, 36, 30
    c = cavity(pkg, (nx, ny, nz), storage, "march", 21)
    m = pkg.lbm.mesh_box(nx, ny, nz, 1.0, ny / nx, nz / nx, "tanh", 1.5)
    s = pkg.slabs.Slabs(pkg.slabs.Domain(nx, ny, nz, Ra=1e5, Pr=0.71, coords=m, storage=storage), nslabs, kernel="march")
    s.initial()
    s.step(21)
    got = s.macro()
    for k, v in c.macro().items():
        assert np.array_equal(got[k], v), k
    s.close()
    c.close()
