"""The weight gradient of images that don't fill the kernel's 8 x 16 pixel tiles:
an infinity or NaN in the last column or row reaches the taps that use it and no
others (a tap's sum has no terms from pixels outside the image).

Reference: float64 sums over the pixel pairs of each tap; a finite sum of n
products accumulated in FP32 is off by at most n 2^-23 sum |x_i| |dz_i|."""
import numpy as np
import pytest

import unet_oracle as U

pytestmark = pytest.mark.gpu


def taps(x, dz):
    """sum over the pixels p with p and p + offset(tap) inside: (Cout, 9, Cin)"""
    B, H, W, Cin = x.shape
    out = np.zeros((dz.shape[-1], 9, Cin))
    for t in range(9):
        dy, dx = t // 3 - 1, t % 3 - 1
        ys, xs = slice(max(0, -dy), H - max(0, dy)), slice(max(0, -dx), W - max(0, dx))
        yi, xi = slice(max(0, dy), H + min(0, dy)), slice(max(0, dx), W + min(0, dx))
        a, b = dz[:, ys, xs].reshape(-1, dz.shape[-1]), x[:, yi, xi].reshape(-1, Cin)
        if len(a):
            with np.errstate(invalid="ignore"):
                out[:, t] = (a[:, :, None] * b[:, None, :]).sum(0)
    return out


# W and H on both sides of a tile's 8 columns, of its 16 rows and of the two rows a step takes; one column, one row;
# several tiles a share, ragged ones among them
@pytest.mark.parametrize("B,H,W,Cin,Cout", [(1, 1, 1, 32, 8), (1, 7, 1, 32, 8), (1, 1, 7, 32, 8), (2, 2, 2, 64, 32),
                                            (2, 5, 5, 32, 40), (1, 3, 8, 32, 32), (1, 16, 13, 32, 8), (1, 17, 9, 64, 16),
                                            (1, 33, 24, 32, 32), (1, 4, 16, 32, 8), (60, 6, 15, 32, 136)])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
def test_infinities_stay_in_their_taps(pkg, B, H, W, Cin, Cout, bad):
    import torch
    lib = pkg.surrogate.nn()
    rng = np.random.default_rng(B * H * W + Cin + Cout)
    x = U.bf16_round(rng.normal(size=(B, H, W, Cin)))
    dz = U.bf16_round(rng.uniform(0.5, 2.0, size=(B, H, W, Cout)) * rng.choice([-1.0, 1.0], size=(B, H, W, Cout)))
    for c, (r, q) in enumerate([(H - 1, W - 1), (0, W - 1), (H - 1, 0), (H // 2, W // 2)]):
        x[c % B, r, q, c] = bad
    xd, zd = (torch.from_numpy(a.astype(np.float32)).cuda().bfloat16() for a in (x, dz))
    n = lib.lbm_nn_wgrad_workspace(B, H, W, Cin, Cout)
    ws = torch.empty(n, device="cuda")
    dw = torch.empty(Cout * 9 * Cin, device="cuda")
    pkg.surrogate.timeouts(reset=True)
    assert lib.lbm_nn_conv3x3_wgrad(zd.data_ptr(), xd.data_ptr(), Cin, 0, B, H, W, Cin, Cout, ws.data_ptr(), n,
                                    dw.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert pkg.surrogate.timeouts(reset=True) == 0
    got = dw.cpu().numpy().astype(np.float64).reshape(Cout, 9, Cin)
    ref = taps(x, dz)
    ok = np.isfinite(ref)
    assert not ok.all()
    assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.array_equal(got[~ok & ~np.isnan(ref)], ref[~ok & ~np.isnan(ref)])
    size = taps(np.where(np.isfinite(x), np.abs(x), 0.0), np.abs(dz))
    assert (np.abs(got - ref)[ok] <= (B * H * W * 2.0 ** -23 * size)[ok]).all()
