"""A convolution or weight gradient whose bounded wait runs out must not leave
an earlier call's values standing as its result.  The wait limit is set so
short that no copy can land in time; the kernels then drain their copies and
return, and the context stays usable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def short_waits(pkg):
    S = pkg.surrogate
    S.timeouts(reset=True)
    yield lambda on: S.set_wait_limit(1 if on else 0)
    S.set_wait_limit(0)
    S.timeouts(reset=True)


# images of one tile and less, ragged ones, several chunks (more than a block's stages) and blocks
@pytest.mark.parametrize("B,R", [(1, 16), (2, 40), (3, 64)])
def test_timed_out_passes_give_nan_not_earlier_values(pkg, short_waits, B, R):
    import torch
    S = pkg.surrogate
    net = S.Net(R=R, seed=3)
    rng = np.random.default_rng(R)
    xs = [torch.from_numpy(rng.normal(size=(B, R, R, S.IN_CH)).astype(np.float32)).cuda().bfloat16() for _ in range(2)]
    tgt = torch.zeros(B * R * R, S.OUT_CH, device="cuda")

    def passes(x):
        y = net.forward(x)
        net.loss(tgt, B)
        net.backward(B)
        torch.cuda.synchronize()
        return y.cpu().numpy().copy(), net.get_params("grad")

    first, other = passes(xs[0]), passes(xs[1])
    net.check()
    short_waits(True)
    y, g = passes(xs[0])
    short_waits(False)
    with pytest.raises(pkg.LBMError) as e:
        net.check()
    assert e.value.status == -5
    # what is not NaN is the answer for this input, not the other one left from the call before
    ok = ~np.isnan(y)
    assert not ok.all() and np.array_equal(y[ok], first[0][ok])
    for name in g:
        for k in range(2):
            ok = ~np.isnan(g[name][k])
            assert np.array_equal(g[name][k][ok], first[1][name][k][ok]), (name, k)
        assert not ok.all() or name == "head", name
    # the counter was taken, and the network works as before
    net.check()
    for x, want in zip(xs, (first, other)):
        y, g = passes(x)
        net.check()
        assert np.array_equal(y, want[0])
        for name in g:
            assert all(np.array_equal(a, b) for a, b in zip(g[name], want[1][name]))


def test_predicted_images_report_a_timeout(pkg, short_waits):
    W = pkg.warmstart.WarmStart(R=16, seed=1)
    X = np.random.default_rng(5).normal(size=(3, 16, 16, 8)).astype(np.float32)
    want = W.predict_images(X)
    short_waits(True)
    with pytest.raises(pkg.LBMError):
        W.predict_images(X)
    short_waits(False)
    assert np.array_equal(W.predict_images(X), want)
