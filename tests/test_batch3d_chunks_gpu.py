"""The 3D batch's work lists: one chunk of a tile column a block where that keeps
the blocks busy, equal contiguous shares elsewhere; a member has the bits of the
same cavity alone whichever it is, and after members have left the list."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# FP64 (296 blocks): one chunk a column, several of unlike length, idle blocks (shares), more columns than blocks
# (shares); FP32 (592) cuts the first three into more; a grid of the caller's
@pytest.mark.parametrize("storage", ["f64", "f32"])
@pytest.mark.parametrize("shapes,nblocks", [([(64, 64, 20)] * 8, 0), ([(40, 24, 33), (33, 12, 50), (96, 40, 7)], 0),
                                            ([(80, 80, 12)] * 3, 0), ([(96, 96, 5)] * 5, 0),
                                            ([(40, 24, 33), (32, 20, 9)], 37)])
def test_members_match_single_cavities(pkg, storage, shapes, nblocks):
    specs = [dict(nx=a, ny=b, nz=c, Ra=1e4, coords=pkg.mesh_box(a, b, c, 1.0, b / a, c / a, "tanh", 1.2))
             for a, b, c in shapes]
    b = pkg.Batch(3, specs, storage=storage)
    if nblocks:
        b.set_option("nblocks", nblocks)
    b.initial()
    singles = []
    for s, sh in zip(specs, shapes):
        c = pkg.Cavity(3, *sh, Ra=1e4, coords=s["coords"], storage=storage, kernel="direct")
        c.initial()
        singles.append(c)
    mask = np.arange(len(shapes)) % 2 == 0
    b.step(5)
    b.run_masked(mask, 4, 2, 0.0)
    for k, c in enumerate(singles):
        c.step(5)
        if mask[k]:
            c.step(4)
    for m, c in zip(b.members, singles):
        for x, y in zip(m.populations(), c.populations()):
            assert np.array_equal(x, y)
        c.close()
    b.close()
