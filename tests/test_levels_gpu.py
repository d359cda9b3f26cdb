"""GPU tests of the fast build's kernels that advance several time steps per
launch: against the oracle at the drop-in tolerance, and bit for bit against
the same run made of single steps (the node arithmetic has explicit rounding,
so how iterations are grouped into launches must not show)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# edges of strips (64 / 128 columns), of the windows at the walls (3 to 5 rows), of segments, and sizes on
# both sides of every rule that picks levels, columns or tiles
SHAPES = [(3, 3), (4, 7), (64, 5), (65, 40), (130, 9), (129, 61), (48, 40), (257, 37), (200, 300)]


def make(pkg, shape, storage="f64", kernel="auto"):
    nx, ny = shape
    co = pkg.mesh_box(nx, ny, 0, 1.0, ny / nx, 1.0, "tanh", 1.3)
    c = pkg.Cavity(2, nx, ny, Ra=1e4, Pr=0.9, coords=co, storage=storage, kernel=kernel)
    y, x = np.meshgrid((np.arange(ny) + 0.5) / ny, (np.arange(nx) + 0.5) / nx, indexing="ij")
    f = (1.0 + 1e-3 * x * y, 0.01 * np.sin(np.pi * x) * np.sin(2 * np.pi * y), -0.01 * np.sin(np.pi * x) * y,
         None, 1.0 - x + 0.05 * np.sin(np.pi * y))
    c.init_equilibrium(*f)
    return c, co, f


@pytest.mark.parametrize("kernel", ["auto", "march"])
@pytest.mark.parametrize("shape", SHAPES)
def test_many_steps_match_oracle(pkg, ora, shape, kernel):
    c, co, f = make(pkg, shape, kernel=kernel)
    o = ora.Oracle(2, *shape, x=co.x, y=co.y, dt=co.dt, length_LB=co.length_LB, Ra=1e4, Pr=0.9)
    o.set_macro(*f)
    for n in (23, 40):
        c.step(n)
        o.step(n)
    got = c.populations()
    for name, a in zip("fg", got):
        ref = o.pops(name)
        assert np.abs(a - ref).max() <= 1e-12 * np.abs(ref).max(), name
    for k, v in c.macro().items():
        assert np.abs(v - o.field(k)).max() <= 1e-12, k
    c.close()


@pytest.mark.parametrize("storage", ["f64", "f32"])
@pytest.mark.parametrize("shape", SHAPES + [(700, 760), (1100, 1000)])
def test_grouping_of_steps_does_not_show(pkg, shape, storage):
    out = []
    for kernel, calls in (("direct", [38]), ("auto", [38]), ("march", [38]), ("auto", [1] * 5 + [17, 9, 7])):
        c, _, _ = make(pkg, shape, storage, kernel)
        for n in calls:
            c.step(n)
        out.append((c.macro(), c.populations()))
        c.close()
    for m, p in out[1:]:
        assert np.array_equal(p[0], out[0][1][0]) and np.array_equal(p[1], out[0][1][1])
        for k in m:
            assert np.array_equal(m[k], out[0][0][k]), k


@pytest.mark.parametrize("storage", ["f64", "f32"])
@pytest.mark.parametrize("tile", [32, 64, 128])
def test_batch_members_match_single_cavities(pkg, storage, tile):
    shapes = [(64, 70), (96, 200), (3, 5), (150, 33), (300, 90)]
    specs = [{"nx": a, "ny": b, "Ra": 1e4, "Pr": 0.9, "coords": pkg.mesh_box(a, b, 0, 1.0, b / a, 1.0, "tanh", 1.3)}
             for a, b in shapes]
    b = pkg.Batch(2, specs, storage=storage)
    b.set_option("tile", tile)
    singles = []
    for m, sh in zip(b.members, shapes):
        c, _, f = make(pkg, sh, storage, "direct")
        m.init_equilibrium(*f)
        singles.append(c)
    for n in (27, 4, 1, 16):
        b.step(n)
        for c in singles:
            c.step(n)
    for m, c in zip(b.members, singles):
        for x, y in zip(m.populations(), c.populations()):
            assert np.array_equal(x, y)
        c.close()
    b.close()
