"""GPU tests of how the fast build's 2D march splits a call's iterations into
launches of 4, 2 and 1 steps, each with a grid and plan of its own: few
launches, and the bits of single direct-load steps whatever the split."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make(pkg, shape, storage, kernel="auto"):
    nx, ny = shape
    co = pkg.mesh_box(nx, ny, 0, 1.0, ny / nx, 1.0, "tanh", 1.3)
    c = pkg.Cavity(2, nx, ny, Ra=1e4, Pr=0.9, coords=co, storage=storage, kernel=kernel)
    y, x = np.meshgrid((np.arange(ny) + 0.5) / ny, (np.arange(nx) + 0.5) / nx, indexing="ij")
    f = (1.0 + 1e-3 * x * y, 0.01 * np.sin(np.pi * x) * np.sin(2 * np.pi * y), -0.01 * np.sin(np.pi * x) * y,
         None, 1.0 - x + 0.05 * np.sin(np.pi * y))
    c.init_equilibrium(*f)
    return c, co, f


def same(a, b):
    for x, y in zip(a.populations(), b.populations()):
        assert np.array_equal(x, y)
    m, n = a.macro(), b.macro()
    assert all(np.array_equal(m[k], n[k]) for k in m)


# four levels of 64 columns (from 2^18 to 2^19 nodes), ragged and close to the upper end; two of 128; two of 64
# (FP64 from 2^21 nodes on)
@pytest.mark.parametrize("storage", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(513, 513), (607, 800), (724, 724), (724, 725), (1023, 771), (2055, 1027)])
def test_every_split_gives_the_bits_of_single_steps(pkg, shape, storage):
    a, _, _ = make(pkg, shape, storage)
    d, _, _ = make(pkg, shape, storage, "direct")
    assert a.kernel == "march"
    for n in (23, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 12):
        a.step(n)
        d.step(n)
    same(a, d)
    a.step(70)  # graph replays
    d.step(70)
    same(a, d)
    a.close()
    d.close()


# 1 + launches of n steps without the last one
@pytest.mark.parametrize("shape,counts", [
    ((513, 513), {1: 1, 2: 2, 3: 3, 4: 4, 5: 3, 6: 4, 7: 3, 8: 4, 9: 3, 11: 5, 13: 5, 15: 5, 17: 5}),
    ((1023, 771), {1: 1, 2: 2, 3: 3, 4: 4, 5: 3, 6: 4, 7: 5, 8: 6, 9: 5, 13: 7})])
def test_launches_of_a_call(pkg, shape, counts):
    c, _, _ = make(pkg, shape, "f64")
    c.step(1)
    for n, want in counts.items():
        before = pkg.lib().lbm_kernel_launches()
        c.step(n)
        assert pkg.lib().lbm_kernel_launches() - before == want, n
    c.close()


# four levels; two levels (FP32 batches of 2^21 nodes and more)
@pytest.mark.parametrize("storage", ["f64", "f32"])
@pytest.mark.parametrize("shapes", [[(64, 70), (3, 5), (150, 33), (300, 90)], [(1100, 1000), (1031, 999)]])
@pytest.mark.parametrize("options", [{"tile": 64}, {"tile": 128}, {"tile": 32, "nblocks": 7}, {"tile": 64, "graphs": 0}])
def test_batch_splits_give_the_bits_of_single_steps(pkg, storage, shapes, options):
    specs = [{"nx": a, "ny": b, "Ra": 1e4, "Pr": 0.9, "coords": pkg.mesh_box(a, b, 0, 1.0, b / a, 1.0, "tanh", 1.3)}
             for a, b in shapes]
    b = pkg.Batch(2, specs, storage=storage)
    for k, v in options.items():
        b.set_option(k, v)
    singles = []
    for m, sh in zip(b.members, shapes):
        c, _, f = make(pkg, sh, storage, "direct")
        m.init_equilibrium(*f)
        singles.append(c)
    for n in (27, 2, 3, 5, 6, 7, 8, 9, 10):
        b.step(n)
        for c in singles:
            c.step(n)
    for m, c in zip(b.members, singles):
        same(m, c)
        c.close()
    b.close()
