"""The x1 march's index arithmetic (csrc/xmarch.cuh: tiles, planes, F buffers,
halo lines), restated and checked for many axis lengths: the tiles cover the
lines that carry unknowns once, tiled copies start on 16 bytes, every
shared-memory place that a thread reads or writes lies inside its ring place
(and so inside the allocation), every F that a row reads is written by exactly
one thread, and every p that a row reads lies in the copied plane. No GPU needed."""
import pytest

T2, T3, RING, LEAD = 16, 8, 7, 3
R2, R3 = T2 + 8, T3 + 8 + 2
PSZ = R2 * R3
SS = 3 * PSZ
PLANE = 2 * SS
R2A = T2 + 4
F2N, F3N = R2A * T3 + 16, T2 * (T3 + 4) + 16
FN = 2 * (F2N + F3N)
# places of the x2 / x3 rows by class (csrc/resident_plan.h, fill_res_tables)
PLACES = [(3, 2, 1, 1), (-1, -1, 1, 2), (-2, -1, 1, 2), (-3, -1, 1, 2), (-2, -1, 1, 2),
          (-1, -1, -2, -3), (-2, -1, 1, 1), (-2, -1, 1, 2), (-2, -1, 1, 3)]


def cls(i, n):
    return i if i < 4 else (5 + (n - 1 - i) if i >= n - 4 else 4)


def x_tiles(n, first, width, step):
    end = n - 1
    best, frm = {first: 0}, {}
    for e in range(first + 1, end + 1):
        if e < end and ((e - first) % step or e < 4 or e > n - 4 or e in (5, n - 5)):
            continue
        for a in range(max(first, e - width), e):
            if a in best and best[a] + 1 < best.get(e, 1 << 20):
                best[e], frm[e] = best[a] + 1, a
    if end not in best:
        return None
    b = [end]
    while b[-1] != first:
        b.append(frm[b[-1]])
    return b[::-1]


@pytest.mark.parametrize("n", list(range(9, 70)) + [81, 101, 129, 161])
def test_tiles_cover_the_axis(n):
    for first, width, step in ((1, T2, 4), (1, T3, 1)):
        b = x_tiles(n, first, width, step)
        assert b is not None and b[0] == 1 and b[-1] == n - 1
        assert all(0 < y - x <= width for x, y in zip(b, b[1:]))
        for x in b[1:-1]:
            assert 4 <= x <= n - 4 and x not in (5, n - 5)
        if step == 4:
            assert all((x - 4 + LEAD) % 4 == 0 for x in b[:-1])   # 16-byte start of the copy


@pytest.mark.parametrize("n2, n3", [(9, 9), (10, 9), (11, 13), (14, 12), (17, 17), (18, 23), (33, 33), (41, 21), (38, 27)])
def test_places_stay_in_bounds_and_are_written(n2, n3):
    b2, b3 = x_tiles(n2, 1, T2, 4), x_tiles(n3, 1, T3, 1)
    for a2, e2 in zip(b2, b2[1:]):
        for a3, e3 in zip(b3, b3[1:]):
            f2w, f3w, f2r, f3r = set(), set(), set(), set()
            dummy = 2 * F2N + F3N - 16
            for tid in range(2 * T2 * T3):
                lane, warp = tid & 31, tid >> 5
                side, k2, k3 = lane & 1, lane >> 1, warp
                i2, i3 = a2 + k2, a3 + k3
                own = i2 < e2 and i3 < e3
                o = side * SS + (k3 + 4) * R2 + k2 + 4
                c2, c3 = (cls(i2, n2), cls(i3, n3)) if own else (4, 4)
                p2, p3 = PLACES[c2], PLACES[c3]
                for d in (p2[0], -1, 1, p2[3], R2 * p3[0], -R2, R2, R2 * p3[3]):
                    for comp in range(3):
                        assert 0 <= o + comp * PSZ + d < PLANE
                if own:
                    for d in p2:
                        assert 0 <= k2 + 4 + d < R2
                    for d in p3:
                        assert 0 <= k3 + 4 + d < R3
                f2 = side * F2N + k3 * R2A + k2 + 2 if own else dummy
                f3 = 2 * F2N + side * F3N + (k3 + 2) * T2 + k2 if own else dummy
                r2 = [f2 + d for d in ((p2[0], -1, 1, p2[3]) if own else (0, -1, 1, 0))]
                r3 = [f3 + d for d in ((T2 * p3[0], -T2, T2, T2 * p3[3]) if own else (0, -T2, T2, 0))]
                assert all(0 <= x < FN for x in r2 + r3 + [f2, f3])
                if own:
                    assert f2 not in f2w and f3 not in f3w
                    f2w.add(f2)
                    f3w.add(f3)
                    # a place with a zero coefficient may repeat another; the others must be written
                    f2r.update(f2 + d for d in p2)
                    f3r.update(f3 + T2 * d for d in p3)
                hal = two = False
                h2 = h3 = hf = 0
                if tid < 128:
                    h3 = a3 - 2 + warp if warp < 2 else e3 + warp - 2
                    h2 = i2
                    hal = h2 < e2 and 0 <= h3 < n3
                    hf = 2 * F2N + side * F3N + (h3 - a3 + 2) * T2 + k2
                elif tid < 128 + 8 * T3:
                    k = (tid - 128) >> 1
                    at = k & 3
                    h2 = a2 - 2 + at if at < 2 else e2 + at - 2
                    h3 = a3 + (k >> 2)
                    hal = two = h3 < e3 and 0 <= h2 < n2
                    hf = side * F2N + (h3 - a3) * R2A + h2 - a2 + 2
                if hal:
                    h = side * SS + (h3 - a3 + 4) * R2 + h2 - a2 + 4
                    for d in PLACES[cls(h2, n2)]:
                        assert 0 <= h2 - a2 + 4 + d < R2 and 0 <= h2 + d < n2
                        assert 0 <= h + PSZ + d < PLANE
                    for d in PLACES[cls(h3, n3)]:
                        assert 0 <= h3 - a3 + 4 + d < R3 and 0 <= h3 + d < n3
                        assert 0 <= h + 2 * PSZ + R2 * d < PLANE
                    w = f2w if two else f3w
                    assert 0 <= hf < FN and hf not in w
                    w.add(hf)
            assert f2r <= f2w and f3r <= f3w
            assert dummy not in f2w | f3w | f2r | f3r
