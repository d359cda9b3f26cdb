"""The grid of the fast build's 3D march past 2^20 nodes: whole chunks alone, nine
tenths of the resident blocks (FP64) or all of them; the bits don't depend on it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# FP64, 296 blocks resident: 128 tiles, two chunks fill them; 200, one does not; 64 tiles of few slices; below the
# rule; more tiles than blocks.  FP32, 592: one chunk of 512 tiles; four of 128
@pytest.mark.parametrize("shape,storage,blocks", [((128, 128, 64), "f64", 256), ((160, 160, 41), "f64", 266),
                                                  ((64, 128, 130), "f64", 256), ((128, 128, 63), "f64", 296),
                                                  ((320, 130, 26), "f64", 296), ((256, 256, 16), "f32", 512),
                                                  ((128, 128, 64), "f32", 592)])
def test_blocks_and_bits(pkg, shape, storage, blocks):
    kw = dict(Ra=1e5, grid="tanh", stretch=1.5, storage=storage)
    c = pkg.Cavity(3, *shape, kernel="march", **kw)
    assert c.get_option(pkg.lbm.OPT_NBLOCKS) == blocks
    d = pkg.Cavity(3, *shape, kernel="march", nblocks=301, **kw)
    for x in (c, d):
        x.initial()
        x.step(5)
    for a, b in zip(c.populations(), d.populations()):
        assert np.array_equal(a, b)
    c.close()
    d.close()
