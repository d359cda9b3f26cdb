"""CPU model of what the march kernels' copying thread does after one of its own
waits gave up (csrc/lbm_march2d.cuh, lbm_march3d.cuh): an mbarrier takes no
second arrival while its phase is open, so no copy may go into a slot whose
last copy the thread has not seen land, and the drain waits for exactly the
copies that were issued.  `guard` False is the schedule without that rule."""
import pytest

from test_march3d_slices import need_hi, need_lo

NS2, ZS, NS3 = 4, 3, 2


class Ring:
    """Slots of one ring: a copy may follow another only after that one was seen to land."""

    def __init__(self, slots):
        self.slots, self.open, self.bad = slots, {}, False

    def issue(self, row):
        if self.open.get(row % self.slots) is not None:
            self.bad = True
        self.open[row % self.slots] = row

    def landed(self, row):
        if self.open.get(row % self.slots) == row:
            self.open[row % self.slots] = None


def march2d(ny, ja, jb, T, fail, guard):
    """The copying thread of a segment [ja, jb); its wait number `fail` gives up, and all threads leave the loop at
    the end of the next iteration.  Returns whether a slot was refilled too early."""
    bottom = ja < T
    row_first, row_last = (0 if bottom else ja - T), min(jb + T - 1, ny - 1)
    its = (jb if bottom else jb - ja + 2) + 3 * (T - 1)
    r1 = min(jb - 1 + T - 1, ny - 1)
    ring, nxt, waits, failed_at, stopped = Ring(NS2), row_first, 0, None, False

    def issue_to(hi):
        nonlocal nxt
        while nxt <= hi and not stopped:
            ring.issue(nxt - row_first)
            nxt += 1

    issue_to(min(row_first + NS2 - 1, row_last))
    for it in range(its):
        q, work = it, True
        if bottom:
            stalls = T - 1
            if q < 4 * stalls:
                n, work = 3 * (q // 4) + q % 4, q % 4 != 3
            else:
                n = q - stalls
        else:
            n = ja - T - 1 + q
        work = work and n <= r1
        n0 = n if work else r1 + 1
        if bottom and not work and q < 4 * (T - 1):
            n0 = 3 * (q // 4) + 3
        issue_to(min(n0 - 1 + NS2, row_last))
        if work:
            rows = (0, 1, 2) if n == 0 and bottom else (() if n == ny - 1 else (n + 1,))
            for r in rows:
                if waits == fail:
                    waits += 1
                    failed_at = it if failed_at is None else failed_at
                    stopped = guard
                    break
                waits += 1
                ring.landed(r - row_first)
        if failed_at is not None and it == failed_at + 1:
            break
    return ring.bad


@pytest.mark.parametrize("T", [2, 4])
def test_march2d(T):
    early = 0
    for ny in (3, 5, 9, 17, 40):
        cuts = [0] + list(range(2, ny - 1))
        for ja in cuts:
            for jb in cuts + [ny]:
                if jb - ja < 2:
                    continue
                for fail in range(jb - ja + T + 3):
                    assert not march2d(ny, ja, jb, T, fail, True), (ny, ja, jb, fail)
                    early += march2d(ny, ja, jb, T, fail, False)
    assert early > 0  # the first row's wait at a segment that starts at the wall


def march3d(n, ka, kb, fail, guard):
    z, p = Ring(ZS), Ring(NS3)
    pre_lo, pre_hi = need_lo(ka, n), need_hi(ka, n)
    seg_hi = max(need_hi(kb - 1, n), pre_hi)
    zi, ni = min(seg_hi, max(pre_hi, ka + ZS - 2)), min(kb - 1, ka + NS3 - 2)
    for s in range(pre_lo, zi + 1):
        z.issue(s)
    for s in range(ka, ni + 1):
        p.issue(s)
    waits, ok = 0, True

    def wait(ring, s):
        nonlocal waits, ok
        if ok and waits == fail:
            ok = False
        waits += 1
        if ok:
            ring.landed(s)

    for s in range(pre_lo, ka + 1):
        wait(z, s)
    for m in range(ka, kb):
        if (ok or not guard) and zi < min(seg_hi, m + ZS - 1):
            zi += 1
            z.issue(zi)
        if (ok or not guard) and ni < min(kb - 1, m + NS3 - 1):
            ni += 1
            p.issue(ni)
        for s in range(need_lo(m, n) if m in (0, n - 1) else m + 1, need_hi(m, n) + 1):
            wait(z, s)
        wait(p, m)
        if not ok:
            break
    return z.bad or p.bad


def test_march3d():
    early = 0
    for n in (3, 4, 5, 9, 14):
        for ka in range(n):
            for kb in range(ka + 1, n + 1):
                for fail in range(4 * (kb - ka) + 4):
                    assert not march3d(n, ka, kb, fail, True), (n, ka, kb, fail)
                    early += march3d(n, ka, kb, fail, False)
    assert early > 0  # a wait before the first step, then that step's refill
