"""The network's tiled kernels at the sizes where a tile ends: images smaller
than a pixel tile, one row or column past it, channel counts with a remainder,
strides and addresses that allow no wide stores.

Reference: the float64 oracle on the same bfloat16 operands.  A sum of n products
accumulated in FP32 in any order, truncating or rounding, is off by at most
n 2^-23 sum |x_i| |w_i|; that is the tolerance, element by element."""
import numpy as np
import pytest

import unet_oracle as U

pytestmark = pytest.mark.gpu


def up(torch, a, dtype=None):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda().to(dtype or torch.float32)


def down(t):
    return t.float().cpu().numpy().astype(np.float64)


# (B, H, W): one pixel; a tile exactly; one past it each way; thin; many images far smaller than a tile
@pytest.mark.parametrize("path", [0, 1])
@pytest.mark.parametrize("B,H,W,Cin,Cout", [(1, 1, 1, 32, 8), (2, 16, 8, 32, 32), (2, 17, 9, 64, 40), (1, 33, 7, 96, 96),
                                            (3, 15, 25, 160, 48), (80, 16, 8, 32, 72), (300, 2, 2, 64, 64)])
def test_convolution_tile_edges(pkg, B, H, W, Cin, Cout, path):
    import torch
    S = pkg.surrogate
    lib = S.nn()
    rng = np.random.default_rng(B * H * W + Cin + Cout)
    x = U.bf16_round(rng.normal(size=(B, H, W, Cin + 8)))
    w = U.bf16_round(rng.normal(0, 0.1, size=(Cout, 9, Cin)))
    bias = rng.normal(size=Cout).astype(np.float32).astype(np.float64)
    bf = torch.bfloat16
    xd, wd, bd = up(torch, x, bf), up(torch, w, bf), up(torch, bias)
    S.timeouts(reset=True)
    S.set_tensor_path(path)
    try:
        got = {}
        for pad, off in ((0, 0), (3, 1)):  # wide stores; odd strides and offsets
            z = torch.full((B, H, W, Cout + pad), 7.0, device="cuda")
            a = torch.full((B, H, W, Cout + pad), 7.0, device="cuda", dtype=bf)
            acc = torch.ones((B, H, W, Cout + pad), device="cuda")
            assert lib.lbm_nn_conv3x3(xd.data_ptr(), Cin + 8, 8, wd.data_ptr(), bd.data_ptr(), B, H, W, Cin, Cout,
                                      z.data_ptr(), Cout + pad, off, 0, a.data_ptr(), Cout + pad, off, 1, None) == 0
            assert lib.lbm_nn_conv3x3(xd.data_ptr(), Cin + 8, 8, wd.data_ptr(), None, B, H, W, Cin, Cout,
                                      acc.data_ptr(), Cout + pad, off, 1, None, 0, 0, 0, None) == 0
            torch.cuda.synchronize()
            sl = slice(off, off + Cout)
            keep = [c for c in range(Cout + pad) if not off <= c < off + Cout]
            assert all((down(t)[..., keep] == v).all() for t, v in ((z, 7.0), (a, 7.0), (acc, 1.0)))
            got[pad] = tuple(down(t)[..., sl] for t in (z, a, acc))
    finally:
        S.set_tensor_path(0)
    assert S.timeouts(reset=True) == 0
    for u, v in zip(got[0], got[3]):
        assert np.array_equal(u, v)
    z, a, acc = got[0]
    ref = U.conv3x3(x[..., 8:], w, np.zeros(Cout))
    size = U.conv3x3(np.abs(x[..., 8:]), np.abs(w), np.zeros(Cout))
    tol = (9 * Cin + 2) * 2.0 ** -23
    assert (np.abs(z - (ref + bias)) <= tol * (size + np.abs(bias))).all()
    assert (np.abs(acc - 1.0 - ref) <= tol * (size + 1.0)).all()
    s = U.silu(z)
    assert (np.abs(a - s) <= 2.0 ** -8 * np.abs(s) + 2.0 ** -8 * 2.0 ** -12).all()


# on both sides of the rule between the two kernels: blocks of tcgen05 (1024 / 1025), how full they are
@pytest.mark.parametrize("B,H,W,Cin,Cout", [(1024, 1, 2, 32, 32), (1025, 1, 2, 32, 32), (1030, 3, 1, 64, 72),
                                            (1025, 4, 4, 32, 8), (1025, 3, 5, 32, 8)])
def test_convolution_of_many_small_images(pkg, B, H, W, Cin, Cout):
    import torch
    S = pkg.surrogate
    rng = np.random.default_rng(B + H * W + Cin + Cout)
    x = U.bf16_round(rng.normal(size=(B, H, W, Cin)))
    w = U.bf16_round(rng.normal(0, 0.1, size=(Cout, 9, Cin)))
    xd, wd = up(torch, x, torch.bfloat16), up(torch, w, torch.bfloat16)
    z = torch.full((B, H, W, Cout), 7.0, device="cuda")
    S.timeouts(reset=True)
    assert S.nn().lbm_nn_conv3x3(xd.data_ptr(), Cin, 0, wd.data_ptr(), None, B, H, W, Cin, Cout, z.data_ptr(), Cout, 0, 0,
                                 None, 0, 0, 0, None) == 0
    torch.cuda.synchronize()
    assert S.timeouts(reset=True) == 0
    ref = U.conv3x3(x, w, np.zeros(Cout))
    size = U.conv3x3(np.abs(x), np.abs(w), np.zeros(Cout))
    assert (np.abs(down(z) - ref) <= (9 * Cin + 2) * 2.0 ** -23 * size).all()


@pytest.mark.parametrize("B,H,W,Cin,Cout", [(1, 1, 1, 32, 8), (2, 8, 16, 32, 32), (2, 9, 17, 64, 40), (1, 7, 33, 96, 72),
                                            (5, 24, 31, 32, 64), (40, 3, 2, 64, 32)])
def test_weight_gradient_tile_edges(pkg, B, H, W, Cin, Cout):
    import torch
    lib = pkg.surrogate.nn()
    rng = np.random.default_rng(B * H * W + Cin + Cout)
    x = U.bf16_round(rng.normal(size=(B, H, W, Cin + 8)))
    dz = U.bf16_round(rng.normal(size=(B, H, W, Cout)))
    xd, dzd = up(torch, x, torch.bfloat16), up(torch, dz, torch.bfloat16)
    n = lib.lbm_nn_wgrad_workspace(B, H, W, Cin, Cout)
    ws = torch.full((n,), float("nan"), device="cuda")
    dw = torch.zeros(Cout * 9 * Cin, device="cuda")
    assert lib.lbm_nn_conv3x3_wgrad(dzd.data_ptr(), xd.data_ptr(), Cin + 8, 8, B, H, W, Cin, Cout, ws.data_ptr(), n,
                                    dw.data_ptr(), None) == 0
    torch.cuda.synchronize()
    ref = U.conv3x3_wgrad(dz, x[..., 8:])
    size = U.conv3x3_wgrad(np.abs(dz), np.abs(x[..., 8:]))
    assert (np.abs(down(dw).reshape(ref.shape) - ref) <= B * H * W * 2.0 ** -23 * size).all()


# one full tile; tiles past the image, several blocks of output channels, one with a remainder; many tiles a share
@pytest.mark.parametrize("B,H,W,Cin,Cout,off", [(1, 16, 8, 32, 8, 0), (3, 37, 21, 96, 264, 0), (2, 33, 47, 32, 160, 1),
                                                (20, 64, 64, 32, 32, 0)])
def test_weight_gradient_channel_blocks_and_shares(pkg, B, H, W, Cin, Cout, off):
    import torch
    lib = pkg.surrogate.nn()
    rng = np.random.default_rng(B * H * W + Cin + Cout)
    x = U.bf16_round(rng.normal(size=(B, H, W, Cin)))
    dz = U.bf16_round(rng.normal(size=(B, H, W, Cout)))
    xd, dzd = up(torch, x, torch.bfloat16), up(torch, dz, torch.bfloat16)
    n = lib.lbm_nn_wgrad_workspace(B, H, W, Cin, Cout)
    ws = torch.full((n + off,), float("nan"), device="cuda")
    dw = torch.full((Cout * 9 * Cin + 2 * off + 1,), 7.0, device="cuda")
    pkg.surrogate.timeouts(reset=True)
    assert lib.lbm_nn_conv3x3_wgrad(dzd.data_ptr(), xd.data_ptr(), Cin, 0, B, H, W, Cin, Cout, ws[off:].data_ptr(), n,
                                    dw[off:].data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert pkg.surrogate.timeouts(reset=True) == 0
    ref = U.conv3x3_wgrad(dz, x)
    size = U.conv3x3_wgrad(np.abs(dz), np.abs(x))
    got = down(dw)
    assert (got[:off] == 7.0).all() and (got[off + ref.size:] == 7.0).all()
    assert (np.abs(got[off:off + ref.size].reshape(ref.shape) - ref) <= B * H * W * 2.0 ** -23 * size).all()


# channels: one 16-byte group, more groups than a block has threads, no multiple of 8; an offset that allows no
# wide loads
@pytest.mark.parametrize("P,C,off", [(1, 8, 0), (1000, 32, 0), (4737, 96, 4), (70, 2056, 0), (333, 36, 0), (333, 32, 1)])
def test_silu_backward_with_bias_gradient(pkg, P, C, off):
    import torch
    lib = pkg.surrogate.nn()
    rng = np.random.default_rng(P + C)
    da, z = rng.normal(size=(P, C + off)), rng.normal(0, 3, size=(P, C))
    dad, zd = up(torch, da), up(torch, z)
    n = max(lib.lbm_nn_colsum_workspace(P, C), 1)
    outs = []
    for fused in (True, False):
        ws = torch.full((n,), float("nan"), device="cuda")
        dz = torch.zeros(P, C, device="cuda", dtype=torch.bfloat16)
        db = torch.zeros(C, device="cuda")
        if fused:
            assert lib.lbm_nn_silu_backward_bias(dad.data_ptr(), C + off, off, zd.data_ptr(), P, C, dz.data_ptr(),
                                                 ws.data_ptr(), db.data_ptr(), None) == 0
        else:
            assert lib.lbm_nn_silu_backward(dad.data_ptr(), C + off, off, zd.data_ptr(), P, C, dz.data_ptr(), None) == 0
            assert lib.lbm_nn_colsum(dz.data_ptr(), P, C, ws.data_ptr(), db.data_ptr(), None) == 0
        torch.cuda.synchronize()
        outs.append((down(dz), down(db)))
    assert np.array_equal(outs[0][0], outs[1][0])
    dz = outs[0][0]
    for _, db in outs:
        assert (np.abs(db - dz.sum(0)) <= P * 2.0 ** -23 * np.abs(dz).sum(0)).all()


def test_the_network_as_one_call_is_its_layers(pkg):
    """The forward pass of lbm_nn_unet_forward against the same layers called one by one: the same bits."""
    import torch
    S = pkg.surrogate
    lib = S.nn()
    B, R = 2, 24
    net = S.Net(R=R, seed=3)
    x = torch.randn(B, R, R, S.IN_CH, generator=torch.Generator().manual_seed(1)).cuda().to(torch.bfloat16)
    y = net.forward(x).clone()
    c1, c2, c3, c4 = S.LEVELS
    st = torch.cuda.current_stream().cuda_stream
    t = {}

    def conv(k, v, xs, out, os_, oo):
        name, ci, co = net.table[k]
        o, ob = net.off[name]
        H = v.shape[1]
        z = torch.empty(B, H, H, co, device="cuda")
        assert lib.lbm_nn_conv3x3(v.data_ptr(), xs, 0, net.pb.data_ptr() + 2 * o, net.master.data_ptr() + 4 * ob, B, H, H,
                                  ci, co, z.data_ptr(), co, 0, 0, out.data_ptr(), os_, oo, 1, st) == 0
        return out

    def new(H, c):
        return torch.zeros(B, H, H, c, device="cuda", dtype=torch.bfloat16)

    v, width = x, S.IN_CH
    for e, (c, up) in enumerate(((c1, c2), (c2, c3), (c3, c4))):
        H = R >> e
        t[e] = conv(2 * e + 1, conv(2 * e, v, width, new(H, c), c, 0), c, new(H, up + c), up + c, up)
        v, width = new(H // 2, c), c
        assert lib.lbm_nn_pool2(t[e].data_ptr(), up + c, up, B, H, H, c, v.data_ptr(), c, 0, st) == 0
    v = conv(7, conv(6, v, c3, new(R // 8, c4), c4, 0), c4, new(R // 8, c4), c4, 0)
    for d, (c, up) in enumerate(((c3, c4), (c2, c3), (c1, c2))):
        e = 2 - d
        H = R >> e
        assert lib.lbm_nn_up2(v.data_ptr(), up, 0, B, H // 2, H // 2, up, t[e].data_ptr(), up + c, 0, st) == 0
        v = conv(9 + 2 * d, conv(8 + 2 * d, t[e], up + c, new(H, c), c, 0), c, new(H, c), c, 0)
    o, ob = net.off["head"]
    want = torch.empty_like(y)
    assert lib.lbm_nn_head(v.data_ptr(), c1, 0, net.pb.data_ptr() + 2 * o, net.master.data_ptr() + 4 * ob, B * R * R, c1,
                           S.OUT_CH, want.data_ptr(), st) == 0
    torch.cuda.synchronize()
    assert torch.equal(y, want)
    import ctypes
    bad = ctypes.byref(S._Unet(B=0, R=R, J=3))
    assert lib.lbm_nn_unet_forward(None, st) < 0 and lib.lbm_nn_unet_backward(bad, st) < 0
