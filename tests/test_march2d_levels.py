"""CPU model of the fast build's 2D march (csrc/lbm_march2d.cuh), which
advances T time levels per pass: the schedule of its groups, the input ring,
the rings between the levels, and the shared-memory columns its stencils touch.

Replayed for a segment [ja, jb) of a column of ny rows, exactly as the kernel
runs it:
  * a group reads only ring rows that the level below finished in an earlier
    iteration, and no row being overwritten in the same iteration;
  * every value a node that reaches the output depends on was computed;
  * the input ring refills a slot only after its row's last reader, every copy
    is waited for, and none is left in flight;
  * each output row is produced exactly once;
  * every column index lies in the row box, whose start is 16-byte aligned.
"""
import pytest

NS, WR = 4, 16


def windows(n, ny):
    lo = 0 if n == 0 else (ny - 3 if n == ny - 1 else n - 1)
    return range(lo, lo + 3)


def replay(ny, ja, jb, T):
    bottom = ja < T
    row_first, row_last = (0 if bottom else ja - T), min(jb + T - 1, ny - 1)
    its = (jb if bottom else jb - ja + 2) + 3 * (T - 1)
    r0 = [max(ja - (T - 1 - s), 0) for s in range(T)]
    r1 = [min(jb - 1 + (T - 1 - s), ny - 1) for s in range(T)]
    slot, weights = {}, {}            # input ring: slot -> row; weight ring: index -> row
    landed, nxt = set(), row_first
    ring = [{} for _ in range(T)]     # ring[s]: slot -> (row, complete)
    hist = [None] * T                 # per group: (row of hx or None, rows in hp)
    out = []

    def issue(hi, reading):
        nonlocal nxt
        while nxt <= hi:
            s = (nxt - row_first) % NS
            assert s not in slot or slot[s] in landed, "refilled before it landed"
            assert s not in slot or slot[s] not in reading, ("refilled while read", nxt)
            slot[s] = nxt
            weights[nxt % WR] = nxt
            nxt += 1

    def node_of(s, it):
        q = it - 3 * s
        if q < 0:
            return None, q
        if bottom:
            stalls = T - 1 - s
            if q < 4 * stalls:
                n = 3 * (q // 4) + q % 4
                if q % 4 == 3:
                    return None, q
            else:
                n = q - stalls
        else:
            n = ja - T + s - 1 + q
        return (n if n <= r1[s] else None), q

    issue(min(row_first + NS - 1, row_last), ())
    for it in range(its):
        n0, q0 = node_of(0, it)
        first = n0 if n0 is not None else r1[0] + 1
        if bottom and n0 is None and q0 < 4 * (T - 1):
            first = 3 * (q0 // 4) + 3
        # group 0's reads of this iteration
        reading = ()
        if n0 is not None:
            reading = windows(n0, ny) if (n0 == 0 and bottom) or n0 == ny - 1 else (n0, n0 + 1)
        issue(min(first - 1 + NS, row_last), reading)
        written = [None] * T
        for s in range(T):
            n, _ = node_of(s, it)
            if n is None:
                continue

            def row(r):
                """(held, complete) of a row of the level below."""
                if s == 0:
                    assert slot.get((r - row_first) % NS) == r, ("input row not resident", r)
                    assert r in landed, r
                    return True
                got = ring[s - 1].get(r % 3)
                return got is not None and got[0] == r and got[1]

            lo, hi = n == 0 and bottom, n == ny - 1
            if s == 0:
                for r in ((0, 1, 2) if lo else (() if hi else (n + 1,))):
                    assert row_first <= r <= row_last
                    landed.add(r)
            if lo or hi:
                ok = all(row(r) for r in windows(n, ny))
                if lo:
                    hist[s] = (row(1), row(0) and row(1))
            else:
                prev = hist[s]
                new = row(n + 1)
                ok = prev is not None and prev[1] and new
                hist[s] = (new, prev is not None and prev[0] and new)
            if n >= r0[s]:
                assert ok, ("a needed row was not computed", s, n)
                assert row(n), ("the node's own row", s, n)
                for r in (n,) if (lo or hi) else (n, n + 1):
                    assert weights.get(r % WR) == r, ("weights", s, r)
                if s == T - 1:
                    out.append(n)
                else:
                    written[s] = n
        # writes land at the barrier; readers of the same iteration were checked against the old contents,
        # but a group may run ahead of its reader inside the iteration: the slot must not be one being read
        for s in range(T - 1):
            if written[s] is None:
                continue
            m, _ = node_of(s + 1, it)
            if m is not None:
                used = set(windows(m, ny)) if (m == 0 and bottom) or m == ny - 1 else {m, m + 1}
                # rows a group only passes through before its first node may be stale
                used = {r for r in used if r >= r0[s]}
                assert written[s] % 3 not in {r % 3 for r in used if r != written[s]}, (s, it, written[s], used)
                assert written[s] not in used
            ring[s][written[s] % 3] = (written[s], True)
    assert out == list(range(ja, jb))
    assert nxt == row_last + 1 and landed >= set(range(row_first, row_last + 1))


def cuts_allowed(ny):
    return [c for c in range(2, ny - 1)]


@pytest.mark.parametrize("T", [1, 2, 4])
@pytest.mark.parametrize("ny", [3, 4, 5, 6, 7, 9, 12, 17, 25, 40])
def test_schedule(T, ny):
    starts = [0] + cuts_allowed(ny)
    for ja in starts:
        for jb in cuts_allowed(ny) + [ny]:
            if jb > ja:
                replay(ny, ja, jb, T)


def strips(nx, nt, T, cp):
    def cut(k, n):
        return 0 if k <= 0 else (nx if k >= n else min((k * nx // n + 4) // 8 * 8, (nx - 2) // 2 * 2))
    halo, S = (T - 1 if cp == 1 else T // 2 * 2), max(1, nx // nt)
    while True:
        c = [(cut(k, S), cut(k + 1, S)) for k in range(S)]
        if all(b - a >= 2 and min(b + halo, nx) - max(a - halo, 0) <= nt for a, b in c):
            return c
        S += 1


@pytest.mark.parametrize("T", [1, 2, 4])
@pytest.mark.parametrize("nt", [32, 64, 128])
@pytest.mark.parametrize("cp", [1, 2])
@pytest.mark.parametrize("es", [8, 4])
def test_columns(T, nt, cp, es):
    # nt: columns of a strip (32: a 64-column kernel on narrower strips); cp: columns of a thread
    HX = 16 // es
    cols = max(nt, 64)
    WB = cols + 2 * HX
    for nx in list(range(3, 300)) + [383, 384, 385, 500, 513, 1023, 2048]:
        done = []
        for x0, x1 in strips(nx, nt, T, cp):
            assert 2 <= x1 - x0 <= 128 and x0 % 2 == 0
            xs = max(x0 - (T - 1 if cp == 1 else T // 2 * 2), 0)
            bx0 = (xs - 1 + HX) // HX * HX - HX
            assert (bx0 * es) % 16 == 0 and (WB * es) % 16 == 0 and WB <= 256 and bx0 <= xs - 1
            have = set(range(max(bx0, 0), min(bx0 + WB, nx)))
            for s in range(T):
                lo, hi = max(x0 - (T - 1 - s), 0), min(x1 + (T - 1 - s), nx)
                threads = [c for c in range(xs, xs + cols, cp) if c + cp > lo and c < hi]
                made = set()
                for c in threads:
                    # element pairs are read and stored at even indices: 16 (FP32: 8) byte accesses
                    assert (c - xs) // cp < cols // cp and (cp == 1 or (c - bx0) % 2 == 0)
                    wall = c == 0 or c + cp >= nx
                    for e in range(cp):
                        w = windows(min(c + e, nx - 1), nx) if wall else range(c + e - 1, c + e + 2)
                        assert 0 <= w[0] - bx0 and w[-1] - bx0 < WB, (nx, x0, s, c)
                        if lo <= c + e < hi:
                            assert list(w) == list(windows(c + e, nx)) and set(w) <= have, (nx, x0, s, c)
                            made.add(c + e)
                    assert c - bx0 + cp - 1 < WB
                    if s == T - 1 and cp == 2 and c + 1 < nx:
                        assert x0 <= c and c + 1 < x1  # stored as a pair
                assert made == set(range(lo, hi))
                have = made
            done += range(x0, x1)
        assert done == list(range(nx))
