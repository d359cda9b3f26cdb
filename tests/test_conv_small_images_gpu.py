"""The mma.sync convolution, which takes many images far smaller than a pixel
tile, with everything a call can ask for: bias, SiLU into a bf16 output, an
offset into wider tensors, odd strides, accumulation.

Reference: the float64 oracle on the same bfloat16 operands; a sum of n products
accumulated in FP32 is off by at most n 2^-23 sum |x_i| |w_i|."""
import numpy as np
import pytest

import unet_oracle as U

pytestmark = pytest.mark.gpu


def up(torch, a, dtype=None):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda().to(dtype or torch.float32)


def down(t):
    return t.float().cpu().numpy().astype(np.float64)


# more than 1024 blocks of tcgen05, tiles less than an eighth full: one column, two by two, a ragged last block of
# pixels; 32 channels and fewer (one kernel), more (the other), remainders of both
@pytest.mark.parametrize("B,H,W,Cin,Cout", [(1040, 1, 1, 32, 8), (1100, 2, 2, 64, 32), (1030, 3, 1, 32, 40),
                                            (1025, 2, 7, 96, 72), (600, 2, 2, 32, 136)])
@pytest.mark.parametrize("pad,off", [(0, 0), (3, 1)])
def test_options(pkg, B, H, W, Cin, Cout, pad, off):
    import torch
    S = pkg.surrogate
    lib = S.nn()
    tiles = B * -(-H // 16) * -(-W // 8)
    assert 8 * B * H * W < tiles * 128 and tiles * -(-Cout // 64) > 1024  # the rule that sends the call there
    rng = np.random.default_rng(B * H * W + Cin + Cout)
    x = U.bf16_round(rng.normal(size=(B, H, W, Cin + 8)))
    w = U.bf16_round(rng.normal(0, 0.1, size=(Cout, 9, Cin)))
    bias = rng.normal(size=Cout).astype(np.float32).astype(np.float64)
    bf = torch.bfloat16
    xd, wd, bd = up(torch, x, bf), up(torch, w, bf), up(torch, bias)
    z = torch.full((B, H, W, Cout + pad), 7.0, device="cuda")
    a = torch.full((B, H, W, Cout + pad), 7.0, device="cuda", dtype=bf)
    lin = torch.full((B, H, W, Cout + pad), 7.0, device="cuda", dtype=bf)
    acc = torch.ones((B, H, W, Cout + pad), device="cuda")
    conv = lambda *rest: lib.lbm_nn_conv3x3(xd.data_ptr(), Cin + 8, 8, wd.data_ptr(), *rest, None)  # noqa: E731
    so = (Cout + pad, off)
    assert conv(bd.data_ptr(), B, H, W, Cin, Cout, z.data_ptr(), *so, 0, a.data_ptr(), *so, 1) == 0
    assert conv(None, B, H, W, Cin, Cout, None, 0, 0, 0, lin.data_ptr(), *so, 0) == 0
    assert conv(None, B, H, W, Cin, Cout, acc.data_ptr(), *so, 1, None, 0, 0, 0) == 0
    torch.cuda.synchronize()
    keep = [c for c in range(Cout + pad) if not off <= c < off + Cout]
    assert all((down(t)[..., keep] == v).all() for t, v in ((z, 7.0), (a, 7.0), (lin, 7.0), (acc, 1.0)))
    z, a, lin, acc = (down(t)[..., off:off + Cout] for t in (z, a, lin, acc))
    ref = U.conv3x3(x[..., 8:], w, np.zeros(Cout))
    size = U.conv3x3(np.abs(x[..., 8:]), np.abs(w), np.zeros(Cout))
    tol = (9 * Cin + 2) * 2.0 ** -23
    assert (np.abs(z - (ref + bias)) <= tol * (size + np.abs(bias))).all()
    assert (np.abs(acc - 1.0 - ref) <= tol * (size + 1.0)).all()
    assert (np.abs(lin - ref) <= tol * size + 2.0 ** -8 * np.abs(ref)).all()
    s = U.silu(z)
    assert (np.abs(a - s) <= 2.0 ** -8 * np.abs(s) + 2.0 ** -8 * 2.0 ** -12).all()


def test_both_kernels_agree(pkg):
    # the same call on the kernel the rule picks and, forced, on tcgen05
    import torch
    S = pkg.surrogate
    rng = np.random.default_rng(3)
    B, H, W, Cin, Cout = 1100, 2, 2, 64, 64
    x = U.bf16_round(rng.normal(size=(B, H, W, Cin)))
    w = U.bf16_round(rng.normal(0, 0.1, size=(Cout, 9, Cin)))
    xd, wd = up(torch, x, torch.bfloat16), up(torch, w, torch.bfloat16)
    out = []
    try:
        for path in (0, 1):
            S.set_tensor_path(path)
            z = torch.empty((B, H, W, Cout), device="cuda")
            assert S.nn().lbm_nn_conv3x3(xd.data_ptr(), Cin, 0, wd.data_ptr(), None, B, H, W, Cin, Cout, z.data_ptr(),
                                         Cout, 0, 0, None, 0, 0, 0, None) == 0
            out.append(down(z))
    finally:
        S.set_tensor_path(0)
    size = U.conv3x3(np.abs(x), np.abs(w), np.zeros(Cout))
    assert (np.abs(out[0] - out[1]) <= 2 * (9 * Cin + 2) * 2.0 ** -23 * size).all()
