"""What the network's calls refuse before any device work, on a machine without
a GPU: fake (never dereferenced) but aligned addresses stand in for device
buffers."""
import ctypes

import pytest

ERR_PARAM = -1


def descriptor(pkg, B, R):
    S = pkg.surrogate
    d = S._Unet(B=B, R=R, J=S.OUT_CH)
    off = 0
    for k, (_, ci, co) in enumerate(S.layer_table()):
        d.ch[2 * k], d.ch[2 * k + 1] = ci, co
        d.off[2 * k], d.off[2 * k + 1] = off, off + 9 * ci * co
        off = S._align(off + 9 * ci * co + co)
    d.off[28], d.off[29] = off, off + S.OUT_CH * S.LEVELS[0]
    for k, (name, kind) in enumerate(S._Unet._fields_[6:-1]):
        a = (k + 1) << 30
        if kind is ctypes.c_void_p:
            setattr(d, name, a)
        else:
            for i in range(kind._length_):
                getattr(d, name)[i] = a + (i << 24)
    return d


def test_a_refused_call_raises_the_librarys_error(pkg):
    S = pkg.surrogate
    with pytest.raises(pkg.LBMError, match="path must be 0") as e:
        S.set_tensor_path(7)
    assert e.value.status == ERR_PARAM


# the scratch is set by the weight gradient; by the column sums, of which the calls before them know nothing
@pytest.mark.parametrize("B,R", [(1, 16), (1, 128), (40, 16), (3, 24)])
def test_backward_refuses_a_small_workspace(pkg, B, R):
    S = pkg.surrogate
    lib = S.nn()
    res = [R, R, R // 2, R // 2, R // 4, R // 4, R // 8, R // 8, R // 4, R // 4, R // 2, R // 2, R, R]
    sizes = {"head": lib.lbm_nn_head_workspace(B * R * R, S.LEVELS[0], S.OUT_CH),
             "colsum": max(lib.lbm_nn_colsum_workspace(B * r * r, co) for r, (_, _, co) in zip(res, S.layer_table())),
             "wgrad": max(lib.lbm_nn_wgrad_workspace(B, r, r, ci, co) for r, (_, ci, co) in zip(res, S.layer_table()))}
    d = descriptor(pkg, B, R)
    for n in (0, sizes["head"], sizes["colsum"] - 1, max(sizes.values()) - 1):
        d.ws_elems = n
        assert lib.lbm_nn_unet_backward(ctypes.byref(d), None) == ERR_PARAM, n
        assert "lbm_nn_unet_backward: workspace" in pkg.lib().lbm_last_error().decode()
