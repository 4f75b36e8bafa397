"""CPU check of the cluster-resident interval kernel's pair layout
(cloning-lbm-mpi_gb300/csrc/clbm_temporal.cu).  A band's rows are stored as
pairs of nodes x and x + ceil(W/2), nine two-lane slots per pair; the kernel's
index arithmetic is restated here, and for every node of every band the slots
a gather step reads and writes are decoded and compared with the pull rules'
(own slot where the reference bounces back, else the neighbour's).  Checked as
well: every slot belongs to one node only, every float offset lies in its
band, every node outside the square's interior is updated exactly once, and a
64-bit access covers the two lanes of one pair."""
import pytest

CX = [0, 1, 0, -1, 0, 1, -1, -1, 1]
CY = [0, 0, 1, 0, -1, 1, 1, -1, -1]
OPP = [0, 3, 4, 1, 2, 7, 8, 5, 6]
GENERAL, EDGE, WALL, BOX, PART, INNER, SEAM = range(7)


def bounce(H, box, x, y):
    """slots of (x, y) that bounce back (src/lbm_src/domain_noSlipWalls.cpp:6-22, square.cpp:24-50)"""
    xmin, xmax, ymin, ymax = box
    m = set()
    if y == H - 1:
        m |= {4, 7, 8}
    if y == 0:
        m |= {2, 5, 6}
    inx, iny = xmin < x < xmax, ymin < y < ymax
    if inx and y == ymin:
        m |= {7, 4, 8}
    if inx and y == ymax:
        m |= {5, 2, 6}
    if iny and x == xmin:
        m |= {6, 3, 7}
    if iny and x == xmax:
        m |= {8, 1, 5}
    for xc, yc, k in ((xmin, ymin, 7), (xmin, ymax, 6), (xmax, ymax, 5), (xmax, ymin, 8)):
        if x == xc and y == yc:
            m.add(k)
    return m


def perimeter(box, ylo, yhi):
    xmin, xmax, ymin, ymax = box
    if yhi < ylo:
        return []
    ncol, nin = (2, xmax - xmin - 1) if xmax > xmin else (1, 0)
    n = ncol * (yhi - ylo + 1) + (nin if ylo == ymin else 0) + (nin if yhi == ymax > ymin else 0)
    side, out = ncol * (yhi - ylo + 1), []
    for j in range(n):
        if j < side:
            out.append((xmax if ncol == 2 and j & 1 else xmin, ylo + (j >> 1 if ncol == 2 else j)))
        else:
            q = j - side
            bottom = ylo == ymin and q < nin
            out.append((xmin + 1 + (q - nin if ylo == ymin and not bottom else q), ymin if bottom else ymax))
    return out


def check(W, H, box, rows):
    xmin, xmax, ymin, ymax = box
    Wh, cs = (W + 1) // 2, len(rows)
    row0 = [sum(rows[:b]) for b in range(cs + 1)]
    div = ((1 << 32) + Wh - 1) // Wh
    in_box = lambda x, y: xmin <= x <= xmax and ymin <= y <= ymax  # noqa: E731
    ps = 2 * 3220  # floats per plane
    assert max(rows) * Wh <= 3220
    col = lambda x: 2 * x if x < Wh else 2 * (x - Wh) + 1  # noqa: E731
    solid = lambda x, y: xmin < x < xmax and ymin < y < ymax  # noqa: E731
    owner, updated, counts = {}, {}, [0] * 6

    def decode(b, row, off):
        """(x, y, k) of float offset `off` in row `row` of band b; x = W: the empty lane"""
        assert 0 <= row < rows[b]
        k, r = divmod(row * 2 * Wh + off, ps)
        i, h = divmod(r, 2)
        assert 0 <= k < 9 and i // Wh == row
        return i % Wh + h * Wh, row0[b] + row, k

    def node(x, y, slots):
        """slots[k] = where S(n,k) is read and P(n, opp k) written"""
        assert (x, y) not in updated
        updated[x, y] = True
        m = bounce(H, box, x, y)
        for k in range(9):
            want = (x, y, k) if k in m else ((x - CX[k]) % W, y - CY[k], OPP[k])
            assert slots[k] == want, (x, y, k)
            s = slots[k]
            if not solid(s[0], s[1]):
                assert owner.setdefault(s, (x, y)) == (x, y), (s, x, y)

    odd = W & 1
    on_seam = lambda xh: xh == 0 or xh >= Wh - 1 - odd  # noqa: E731
    for b in range(cs):
        n, ylo, yhi = rows[b] * Wh, max(ymin, row0[b]), min(ymax, row0[b] + rows[b] - 1)
        box_edge = ylo <= yhi and ((ylo == row0[b] and b > 0) or (yhi == row0[b] + rows[b] - 1 and b + 1 < cs))
        for x, y in perimeter(box, ylo, yhi):
            assert in_box(x, y) and not solid(x, y) and row0[b] <= y < row0[b + 1]
            ly, m = y - row0[b], bounce(H, box, x, y)
            C = (b, ly)  # gather step: in A alone, or anywhere in the cluster where the square touches a band edge
            U = (b - 1, rows[b - 1] - 1) if box_edge and ly == 0 else (b, ly - 1)
            D = (b + 1, 0) if box_edge and ly == rows[b] - 1 else (b, ly + 1)
            co, cm, cp = col(x), col(W - 1 if x == 0 else x - 1), col(0 if x == W - 1 else x + 1)
            slots = []
            for k in range(9):
                row, sx = {1: U, 0: C, -1: D}[CY[k]], {1: cm, 0: co, -1: cp}[CX[k]]
                slots.append(decode(*C, co + k * ps) if k in m else decode(*row, sx + OPP[k] * ps))
            assert not any(solid(*s[:2]) for s in slots)  # every slot across the surface bounces back
            node(x, y, slots)

        def pair(c, ly, xh):
            y, o, x1 = row0[b] + ly, 2 * xh, xh + Wh
            if c in (GENERAL, SEAM):
                m0, p0 = col(W - 1 if xh == 0 else xh - 1), col(0 if xh + 1 == W else xh + 1)
                m1 = col(x1 - 1) if x1 < W else o + 1
                p1 = col(0 if x1 + 1 == W else x1 + 1) if x1 < W else o + 1
            else:
                m0, m1, p0, p1 = o - 2, o - 1, o + 2, o + 3
            wb, wt = y == 0 and c in (GENERAL, WALL), y == H - 1 and c in (GENERAL, WALL)
            C = (b, ly)
            U = C if wb else ((b - 1, rows[b - 1] - 1) if ly == 0 and c in (GENERAL, EDGE) else (b, ly - 1))
            D = C if wt else ((b + 1, 0) if ly == rows[b] - 1 and c in (GENERAL, EDGE) else (b, ly + 1))
            at = [(C, o, o + 1), (C, m0 + 3 * ps, m1 + 3 * ps), (U, o + (2 if wb else 4) * ps, o + 1 + (2 if wb else 4) * ps),
                  (C, p0 + ps, p1 + ps), (D, o + (4 if wt else 2) * ps, o + 1 + (4 if wt else 2) * ps),
                  (U, o + 5 * ps, o + 1 + 5 * ps) if wb else (U, m0 + 7 * ps, m1 + 7 * ps),
                  (U, o + 6 * ps, o + 1 + 6 * ps) if wb else (U, p0 + 8 * ps, p1 + 8 * ps),
                  (D, o + 7 * ps, o + 1 + 7 * ps) if wt else (D, p0 + 5 * ps, p1 + 5 * ps),
                  (D, o + 8 * ps, o + 1 + 8 * ps) if wt else (D, m0 + 6 * ps, m1 + 6 * ps)]
            for h, x in ((0, xh), (1, xh + Wh)):
                slots = [decode(*row, (e0, e1)[h]) for row, e0, e1 in at]
                if x >= W:  # the empty lane keeps to its own column
                    assert all(s[0] == W for s in slots)
                elif in_box(x, y):
                    assert c in (GENERAL, SEAM, BOX)  # not written there: a perimeter node, or the interior
                else:
                    node(x, y, slots)
            if c not in (GENERAL, SEAM):
                assert all(e0 % 2 == 0 and e1 == e0 + 1 for _, e0, e1 in at)

        ns = 3 if odd and Wh > 2 else 2
        for j in range(ns * rows[b]):
            ly, s = divmod(j, ns)
            assert on_seam(0 if s == 0 else Wh - s)
            pair(GENERAL if ly in (0, rows[b] - 1) else SEAM, ly, 0 if s == 0 else Wh - s)
        spr = (Wh + 31) // 32
        segs = [(32 * s, Wh) for s in range(spr)]
        if rows[b] > 1:
            segs += [((rows[b] - 1) * Wh + 32 * s, n) for s in range(spr)]
            segs += [(s, n - Wh) for s in range(Wh, n - Wh, 32)]
        for sg, (start, lim) in enumerate(segs):
            lanes = []
            for i in range(start, start + 32):
                ly = i * div >> 32
                assert ly == i // Wh
                p = i - ly * Wh
                lanes.append((i, ly, Wh - 1 if p == 0 else p - 1, i < lim))
            box_ = any(q and (in_box(xh, row0[b] + ly) or in_box(xh + Wh, row0[b] + ly)) for _, ly, xh, q in lanes)
            full = all(q and not on_seam(xh) for _, ly, xh, q in lanes)
            if sg < 2 * spr:
                wall = row0[b] == 0 if sg < spr else row0[b] + rows[b] == H
                c = GENERAL if rows[b] == 1 or box_ else WALL if wall else EDGE
                assert c != EDGE or cs > 1
            else:
                c = BOX if box_ else INNER if full else PART
            counts[c] += 1
            for i, ly, xh, q in lanes:
                if q and not on_seam(xh):
                    if c == INNER:
                        assert i - 1 == ly * Wh + xh
                    pair(c, ly, xh)
    assert len(updated) == sum(not solid(x, y) for x in range(W) for y in range(H))
    return counts


@pytest.mark.parametrize("NW", [8, 16, 24, 32])
def test_deal_covers_every_entry_once(NW):
    """The round robin with one round left out for the warps of the head."""
    for nhead in (0, 1, 5, NW - 1, NW, NW + 3):
        for n in (0, 1, NW - 1, NW, 3 * NW + 2):
            seen = []
            for warp in range(NW):
                if nhead >= NW:
                    q, dq = (warp - nhead) % NW, NW
                else:
                    q = warp - nhead if warp >= nhead else 2 * (NW - nhead) + warp
                    dq = NW - nhead if warp >= nhead else NW
                while q < n:
                    seen.append(q)
                    q, dq = q + dq, NW
            assert sorted(seen) == list(range(n)), (nhead, n)


@pytest.mark.parametrize("W,H,side,xc,yc,rows", [
    (256, 64, 12, 64, 32, [25, 14, 25]), (256, 64, 12, 64, 32, [16] * 4), (200, 50, 8, 50, 25, [12, 8, 6, 12, 12]),
    (96, 23, 5, 30, 9, [5, 5, 5, 4, 4]), (96, 23, 5, 30, 9, [20, 3]), (64, 24, 6, 16, 12, [1, 11, 11, 1]),
    (64, 24, 6, 16, 12, [24]), (97, 33, 6, 24, 16, [17, 16]), (97, 33, 6, 50, 16, [33]), (129, 65, 16, 60, 30, [30, 2, 33]),
    (101, 41, 9, 95, 20, [41]), (65, 20, 5, 2, 10, [9, 11]), (33, 17, 4, 8, 8, [17]), (7, 9, 2, 3, 4, [4, 5]),
    (3, 8, 1, 1, 3, [8]), (400, 100, 20, 100, 50, [12] + [11] * 8), (513, 31, 6, 255, 15, [8, 8, 8, 7]),
])
def test_pair_slots_follow_the_pull_rules(W, H, side, xc, yc, rows):
    xmin, ymin = xc - side // 2, yc - side // 2
    counts = check(W, H, (xmin, xmin + side, ymin, ymin + side), rows)
    Wh = (W + 1) // 2
    spr = (Wh + 31) // 32
    assert sum(counts) == sum(spr if r == 1 else 2 * spr + ((r - 2) * Wh + 31) // 32 for r in rows)
