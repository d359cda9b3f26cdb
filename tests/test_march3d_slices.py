"""CPU model of the fast build's 3D march along z (csrc/lbm_march3d.cuh): the
schedule of copies into the slice rings and the slices a thread carries.

Every segment is replayed in both directions with symbolic slices.  Checked: a
slice is resident, and its copy waited for, whenever it is read; a slot is
refilled only after every read of what it held, with a block barrier between;
each output combines exactly its window's slices, lowest first, with the
weights of its own row."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from test_march_schedule import library_plan, need_hi, need_lo  # noqa: E402

ZS, NS = 3, 2


def window(k, n):
    lo = 0 if k == 0 else (n - 3 if k == n - 1 else k - 1)
    return (lo, lo + 1, lo + 2)


def replay_segment(n, z0, z1, rev):
    ka, kb = (n - z1, n - z0) if rev else (z0, z1)
    z, zwait, zread = {}, set(), {}      # slot -> slice; slices waited for; slot -> barrier count of the last read
    p, pread = {}, {}
    state = {"bar": 0}
    real = (lambda s: n - 1 - s) if rev else (lambda s: s)

    def issue(ring, reads, nslots, s):
        assert 0 <= s < n
        assert reads.get(s % nslots, -1) < state["bar"], ("slot refilled before a barrier", s)
        ring[s % nslots] = s

    def value(s):
        assert z.get(s % ZS) == s and s in zwait, ("slice not resident", s)
        zread[s % ZS] = state["bar"]
        return real(s)

    pre_lo, pre_hi = need_lo(ka, n), need_hi(ka, n)
    seg_hi = max(need_hi(kb - 1, n), pre_hi)
    zissued, nissued = min(seg_hi, max(pre_hi, ka + ZS - 2)), min(kb - 1, ka + NS - 2)
    for s in range(pre_lo, zissued + 1):
        issue(z, zread, ZS, s)
    for s in range(ka, nissued + 1):
        issue(p, pread, NS, s)
    zwait.update(range(pre_lo, ka + 1))
    va = value(ka - 1) if ka > 0 else None
    vb = value(ka)
    state["bar"] += 1
    done = []
    for m in range(ka, kb):
        k = real(m)
        if zissued < min(seg_hi, m + ZS - 1):
            zissued += 1
            issue(z, zread, ZS, zissued)
        if nissued < min(kb - 1, m + NS - 1):
            nissued += 1
            issue(p, pread, NS, nissued)
        end = m in (0, n - 1)
        zwait.update(range(need_lo(m, n) if end else m + 1, need_hi(m, n) + 1))
        vc = value(m + 1) if m < n - 1 else None
        assert p[m % NS] == m
        pread[m % NS] = state["bar"]
        if not end:
            o = (va, vb, vc)
            w = (2, 1, 0) if rev else (0, 1, 2)      # the weights' indices, slice behind first
            assert tuple(sorted(zip(o, w))) == tuple(zip(window(k, n), (0, 1, 2)))
        else:
            x = value(2 if m == 0 else n - 3)
            mid = vc if m == 0 else va
            o = (vb, mid, x) if k == 0 else (x, mid, vb)
            assert o == window(k, n), (n, z0, z1, rev, k, o)
        assert value(m) == k                         # wall nodes read the centre slice
        done.append(k)
        va, vb = vb, vc
        state["bar"] += 1
    assert zissued == seg_hi and set(range(pre_lo, seg_hi + 1)) <= zwait
    assert sorted(done) == list(range(z0, z1))


@pytest.mark.parametrize("n", [3, 4, 5, 6, 7, 13])
def test_every_segment_in_both_directions(n):
    for z0 in range(n):
        for z1 in range(z0 + 1, n + 1):
            for rev in (False, True):
                replay_segment(n, z0, z1, rev)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("ntiles,nz,grid", [(128, 128, 296), (150, 125, 296), (26, 47, 296), (3, 3, 148), (2, 20, 7)])
def test_plans_cover_every_slice_once(ntiles, nz, grid, kind):
    seen = set()
    for segs in library_plan(ntiles, nz, grid, kind):
        for t, z0, z1 in segs:
            for rev in (False, True):
                replay_segment(nz, z0, z1, rev)
            for k in range(z0, z1):
                assert (t, k) not in seen
                seen.add((t, k))
    assert len(seen) == ntiles * nz
