"""The fast build's march kernels bound every wait for their TMA copies: one that
runs out makes the step report LBM_ERR_TIMEOUT (the kernel stops issuing, drains
its copies and returns), and with the limit restored a re-initialised run has
the bits of an untouched one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 2D: one level only (two steps), four levels, two levels of 128 columns; 3D whole and ragged tiles
CASES = [(2, (256, 48, 1), 2), (2, (520, 510, 1), 17), (2, (900, 700, 1), 9), (3, (64, 24, 16), 4), (3, (40, 34, 20), 5)]


@pytest.mark.parametrize("storage", ["f64", "f32"])
@pytest.mark.parametrize("dim,shape,steps", CASES)
def test_single_cavity(pkg, dim, shape, steps, storage):
    L = pkg.lbm

    def run(c):
        c.initial()
        c.step(steps)
        return c.populations()

    kw = dict(grid="tanh", stretch=1.5, storage=storage, kernel="march")
    ref = pkg.Cavity(dim, *shape, **kw)
    want = run(ref)
    ref.close()
    c = pkg.Cavity(dim, *shape, **kw)
    c.initial()
    c.set_option(L.OPT_WAIT_LIMIT, 1)
    try:
        with pytest.raises(pkg.LBMError) as e:
            c.step(steps)
            c.synchronize()
        assert e.value.status == -5 and "bounded wait" in str(e.value)
    finally:
        c.set_option(L.OPT_WAIT_LIMIT, 0)
    c.synchronize()  # the flag was cleared when it was reported
    got = run(c)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
    c.close()


@pytest.mark.parametrize("dim,shape", [(2, (200, 150, 1)), (3, (40, 32, 20))])
def test_batch(pkg, dim, shape):
    L = pkg.lbm
    specs = [dict(nx=shape[0], ny=shape[1], nz=shape[2])] * 3

    def run(b):
        b.initial()
        b.step(17)
        b.synchronize()
        return [m.populations() for m in b.members]

    ref = pkg.Batch(dim, specs)
    want = run(ref)
    ref.close()
    b = pkg.Batch(dim, specs)
    b.initial()
    b.members[0].set_option(L.OPT_WAIT_LIMIT, 1)  # for every kernel on the device
    try:
        with pytest.raises(pkg.LBMError) as e:
            b.step(17)
            b.synchronize()
        assert e.value.status == -5
    finally:
        b.members[0].set_option(L.OPT_WAIT_LIMIT, 0)
    b.synchronize()
    for got, w in zip(run(b), want):
        assert all(np.array_equal(x, y) for x, y in zip(got, w))
    b.close()
