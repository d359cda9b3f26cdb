"""LBM_OPT_KERNEL = 2 is the march kernel for small 2D domains too, where the
automatic choice advances tiles in shared memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# sizes of tests/test_levels_gpu.py, all of which the automatic choice would give tiles: edges of strips, of the
# windows at the walls and of segments
SHAPES = [(3, 3), (4, 7), (64, 5), (65, 40), (130, 9), (129, 61), (48, 40), (257, 37), (200, 300), (300, 250)]


def make(pkg, shape, storage, kernel):
    nx, ny = shape
    co = pkg.mesh_box(nx, ny, 0, 1.0, ny / nx, 1.0, "tanh", 1.3)
    c = pkg.Cavity(2, nx, ny, Ra=1e4, Pr=0.9, coords=co, storage=storage, kernel=kernel)
    y, x = np.meshgrid((np.arange(ny) + 0.5) / ny, (np.arange(nx) + 0.5) / nx, indexing="ij")
    c.init_equilibrium(1.0 + 1e-3 * x * y, 0.01 * np.sin(np.pi * x) * np.sin(2 * np.pi * y),
                       -0.01 * np.sin(np.pi * x) * y, None, 1.0 - x + 0.05 * np.sin(np.pi * y))
    return c


@pytest.mark.parametrize("storage", ["f64", "f32"])
@pytest.mark.parametrize("shape", SHAPES)
def test_march_of_several_levels_gives_the_bits_of_single_steps(pkg, shape, storage):
    a, d = make(pkg, shape, storage, "march"), make(pkg, shape, storage, "direct")
    for n in (38, 7, 6, 5):
        a.step(n)
        d.step(n)
    for x, y in zip(a.populations(), d.populations()):
        assert np.array_equal(x, y)
    a.close()
    d.close()


def test_launches_are_the_march_kernels(pkg):
    # 16 steps as four launches of four levels, then the last one; tiles of a domain this small take eight steps each
    counts = {}
    for shape in [(12, 10), (20, 16)]:
        for kernel in ("auto", "march"):
            c = make(pkg, shape, "f64", kernel)
            c.step(1)
            before = pkg.lib().lbm_kernel_launches()
            c.step(17)
            counts[shape, kernel] = pkg.lib().lbm_kernel_launches() - before
            c.close()
    assert all(n == 5 for (_, kernel), n in counts.items() if kernel == "march"), counts
    assert any(n != 5 for (_, kernel), n in counts.items() if kernel == "auto"), counts
