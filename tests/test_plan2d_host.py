"""The library's plans of the 2D launches of several steps (host code): every
row of every column in one segment, strips that fit the kernel's rows with
their halo, no wall row by itself, segments the kernel's schedule runs (the CPU
model of test_march2d_levels), and tiles whose patches fit what is reserved."""
import ctypes

import pytest

from test_march2d_levels import replay

ERR_PARAM = -1


def march_plan(pkg, nx, ny, columns, levels, nblocks):
    fn = pkg.lib().lbm_march_plan2d
    n, used = ctypes.c_int32(0), ctypes.c_int32()
    assert fn(nx, ny, columns, levels, nblocks, ctypes.byref(n), None, None, ctypes.byref(used)) == 0
    segs, off = (ctypes.c_int32 * (4 * n.value))(), (ctypes.c_int32 * (used.value + 1))()
    assert fn(nx, ny, columns, levels, nblocks, ctypes.byref(n), segs, off, ctypes.byref(used)) == 0
    return [tuple(segs[4 * k:4 * k + 4]) for k in range(n.value)], list(off)


SIZES = [(3, 3), (4, 7), (5, 4), (31, 33), (64, 5), (65, 40), (129, 61), (250, 9), (513, 513), (724, 725), (1023, 771),
         (2055, 127), (40, 3000)]


@pytest.mark.parametrize("levels", [2, 4])
@pytest.mark.parametrize("columns", [32, 64, 128])
@pytest.mark.parametrize("nblocks", [1, 7, 148, 296, 1776])
def test_march_plan(pkg, levels, columns, nblocks):
    replayed = set()
    for nx, ny in SIZES:
        segs, off = march_plan(pkg, nx, ny, columns, levels, nblocks)
        assert off[0] == 0 and off[-1] == len(segs) and all(a < b for a, b in zip(off, off[1:]))
        assert len(off) - 1 <= nblocks
        strips = {}
        for x0, w, ja, jb in segs:
            assert 0 <= ja < jb <= ny
            strips.setdefault((x0, w), []).append((ja, jb))
        done = 0
        for x0, w in sorted(strips):
            assert x0 == done and w >= 2 and (x0 % 8 == 0 or x0 + w == nx)
            done = x0 + w
            assert min(done + levels - 1, nx) - max(x0 - (levels - 1), 0) <= columns
            rows = sorted(strips[x0, w])
            assert rows[0][0] == 0 and rows[-1][1] == ny and all(a[1] == b[0] for a, b in zip(rows, rows[1:]))
            for ja, jb in rows:
                assert jb >= 2 and ja <= ny - 2
                key = (min(ja, 12), jb - ja if jb - ja < 40 else 40, min(ny - jb, 12))
                if ny < 200 and key not in replayed:
                    replayed.add(key)
                    replay(ny, ja, jb, levels)
        assert done == nx
        # the shares: no block has more iterations than twice the mean and a segment's overhead
        cost = [sum(jb - ja + 3 * levels - 1 for _, _, ja, jb in segs[a:b]) for a, b in zip(off, off[1:])]
        total = sum(jb - ja for _, _, ja, jb in segs) + (3 * levels - 1) * len(strips)
        assert max(cost) <= max(2 * total / nblocks, 4) + 2 * (3 * levels - 1) + 4


def cut(a, nt, n, m):
    if a <= 0:
        return 0
    return n if a >= nt else min((a * n // nt + m // 2) // m * m, n - 2)


@pytest.mark.parametrize("esize", [8, 4])
@pytest.mark.parametrize("sms", [148, 132, 20])
def test_tile_plan(pkg, esize, sms):
    plan = (ctypes.c_int32 * 6)()
    some = 0
    for nx in (3, 4, 9, 16, 17, 48, 65, 100, 128, 200, 257, 300, 511):
        for ny in (3, 5, 40, 64, 127, 180, 300, 512, 2000):
            if nx * ny > 1 << 18:
                continue
            assert pkg.lib().lbm_tile_plan2d(nx, ny, esize, sms, plan) == 0
            ntx, nty, T, en, threads, smem = plan
            assert 0 <= T <= 8
            if T < 2:
                continue
            some += 1
            assert threads % 32 == 0 and 64 <= threads <= 512 and smem <= 227 * 1024
            for t in range(1, T + 1):  # a launch may take fewer steps
                for a in range(ntx):
                    X0, X1 = cut(a, ntx, nx, 8), cut(a + 1, ntx, nx, 8)
                    assert X1 - X0 >= 2
                    ew = min(X1 + t, nx) - max(X0 - t, 0)
                    for b in (0, nty // 2, nty - 1):
                        Y0, Y1 = cut(b, nty, ny, 1), cut(b + 1, nty, ny, 1)
                        assert Y1 - Y0 >= 2
                        eh = min(Y1 + t, ny) - max(Y0 - t, 0)
                        assert ew >= 3 and eh >= 3 and ew * eh <= en
                        assert (2 * en * 15 + (ew + eh) * 7) * esize <= smem
    assert some > 20


def test_bad_arguments(pkg):
    n = ctypes.c_int32(0)
    for bad in ((2, 9, 64, 4, 1), (9, 2, 64, 4, 1), (9, 9, 48, 4, 1), (9, 9, 64, 1, 1), (9, 9, 64, 4, 0)):
        assert pkg.lib().lbm_march_plan2d(*bad, ctypes.byref(n), None, None, None) == ERR_PARAM
    assert pkg.lib().lbm_tile_plan2d(9, 9, 2, 148, (ctypes.c_int32 * 6)()) == ERR_PARAM
    assert pkg.lib().lbm_tile_plan2d(9, 9, 8, 148, None) == ERR_PARAM
