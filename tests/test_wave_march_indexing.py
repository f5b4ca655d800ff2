"""The index arithmetic of the strip kernels (csrc/lb_pair.cuh: wave_march),
restated on the CPU for two and four steps per launch: every staged copy
aligned and in bounds, every shared-memory index within the warp's share, every
level's populations and force those of the level before at the node they stream
from (bounced back at the walls, from the ghost rows of a y-slab), every level's
moments and the last level's state stored once per node.  A value is the code of
what it stands for: (level, population, row, column)."""
import numpy as np
import pytest

CX = [0, 1, 0, -1, 0, 1, -1, -1, 1]
CY = [0, 0, 1, 0, -1, 1, 1, -1, -1]
OPP = [0, 3, 4, 1, 2, 7, 8, 5, 6]
BAD = -1
LANE = np.arange(32)
NEXT = np.minimum(LANE + 1, 31)
SLOTS, STAGE = 7 + 2 * 6, 2 * 9 + 1


def level_cols(s):
    return 2 * (32 - s)


def lag_start(s):
    return sum(SLOTS * level_cols(q) for q in range(1, s + 1))


def code(s, k, y, x, nx):
    """population k (9: the force for the next level) after s steps at (y, x)"""
    return ((s * 10 + k) * 4096 + (y + 2)) * 8192 + np.asarray(x) % nx


class Lag:
    """a warp's rows between the levels, with the floats past them that lanes
    beyond a level's last pair may read"""

    def __init__(self, S):
        self.v = np.full((lag_start(S - 1) + 8 + 3) // 4 * 4, BAD, dtype=np.int64)

    def read(self, i):
        assert i.min() >= 0 and i.max() < len(self.v)
        return self.v[i]


def down(a):
    return np.where(LANE < 31, a[NEXT], a)  # __shfl_down_sync(., 1)


def march(S, fp64, nx, ny, x0, ncols, ya, Hc, glo, ghi, stored):
    D = 1
    vec = 2 if fp64 else 4
    ylo, yhi = (-1 if glo else 0), (ny if ghi else ny - 1)

    def pulled(s, k, y, x):
        """population k streaming into (y, x) after s steps"""
        js = y - CY[k]
        if (js < 0 and not glo) or (js >= ny and not ghi):
            return code(s, OPP[k], y, x, nx)
        return code(s, k, js, x - CX[k], nx)

    def stage(y):
        st = np.full((10, 64), BAD, dtype=np.int64)
        if not 0 < y < ny - 1:
            return st
        for lane in range(32 if fp64 else 16):
            cq = vec * lane
            if cq >= ncols + 2 * S:
                continue
            col = (x0 - S + cq + nx) % nx
            assert x0 - S + nx >= 0 and col % vec == 0 and col + vec <= nx and cq + vec <= 64
            for k in range(9):
                assert 0 <= y - CY[k] < ny
                st[k, cq:cq + vec] = code(0, k, y - CY[k], col + np.arange(vec), nx)
            st[9, cq:cq + vec] = code(0, 9, y, col + np.arange(vec), nx)
        return st

    def collide(s, y, f, F):
        """a level's results, where all its inputs are what they have to be"""
        col = x0 - (S - s) + 2 * LANE
        good = np.ones((2, 32), bool)
        for c in range(2):
            for k in range(9):
                good[c] &= f[k][c] == pulled(s - 1, k, y, col + c)
            good[c] &= F[c] == code(s - 1, 9, y, col + c, nx)
        inside = ylo <= y <= yhi
        out = [[np.where(good[c] & inside, code(s, k, y, col + c, nx), BAD) for c in range(2)] for k in range(10)]
        return out[:9], out[9]

    lag = Lag(S)
    nit = Hc + 2 * (S - 1)
    y = ya - (S - 1)
    p0, p1 = 0, 6
    for it in range(nit):
        st = stage(y)
        f, F = [[np.full(32, BAD)] * 2 for _ in range(9)], [np.full(32, BAD)] * 2
        if 0 < y < ny - 1:
            own = lambda i: [st[i][2 * LANE], st[i][2 * LANE + 1]]
            nxt = lambda i: [st[i][2 * NEXT], st[i][2 * NEXT + 1]]
            mid = lambda i: [st[i][2 * LANE + 1], st[i][2 * NEXT]]
            f = [own(k) if CX[k] == 1 else (nxt(k) if CX[k] == -1 else mid(k)) for k in range(9)]
            F = mid(9)
        elif ylo <= y <= yhi:
            col = x0 - (S - 1) + 2 * LANE
            assert (col + nx).min() >= 0
            f = [[pulled(0, k, y, col + c) for c in range(2)] for k in range(9)]
            F = [code(0, 9, y, col + c, nx) for c in range(2)]
        f, F = collide(1, y, f, F)
        for s in range(1, S + 1):
            off, yr = S - s, y - (s - 1)
            if 0 <= yr - ya < Hc:
                c = 2 * LANE - off + (off & 1)
                ok = (c >= 0) & (c < ncols)
                for k in range(10) if s == S else (9,):
                    a = F if k == 9 else f[k]
                    b = [a[1], down(a[0])] if off & 1 else a
                    for q in range(2):
                        want = code(s, k, yr, x0 + c + q, nx)
                        assert (b[q][ok] == want[ok]).all(), (S, s, k, it)
                for cc in c[ok]:
                    assert 0 <= yr < ny and cc + 1 < ncols
                    for q in range(2):
                        x = x0 + cc + q
                        x = x - nx if x >= nx else x
                        assert 0 <= x < nx
                        key = (s, yr, x)
                        stored[key] = stored.get(key, 0) + 1
            if s == S:
                break
            yn = yr - 1
            lo, hi = yn == 0 and not glo, yn == ny - 1 and not ghi
            CW = level_cols(s)
            w0 = lag_start(s - 1)
            w1, wp = w0 + (7 + p0) * CW, w0 + (7 + p1) * CW
            own = lambda q, i: [lag.read(q + i * CW + 2 * LANE), lag.read(q + i * CW + 2 * LANE + 1)]
            nxt = lambda q, i: [lag.read(q + i * CW + 2 * NEXT), lag.read(q + i * CW + 2 * NEXT + 1)]
            mid = lambda q, i: [lag.read(q + i * CW + 2 * LANE + 1), lag.read(q + i * CW + 2 * NEXT)]
            a0, a1, a3, Fn = mid(w0, 0), own(w0, 1), nxt(w0, 2), mid(w0, 6)
            a2, a5, a6 = mid(w1, 0), own(w1, 1), nxt(w1, 2)
            if lo:
                a5, a6 = mid(w1, 1), mid(w1, 2)

            def put(q, i, a):
                lanes = LANE[2 * LANE < CW]
                at = q + i * CW + 2 * lanes
                assert at.max() + 1 < lag_start(s)
                lag.v[at], lag.v[at + 1] = a[0][lanes], a[1][lanes]

            put(w0, 0, f[0]), put(w0, 1, f[1]), put(w0, 2, f[3]), put(w0, 6, F)
            put(w1, 0, f[2]), put(w1, 1, f[5]), put(w1, 2, f[6])
            if yr == 0 and not glo:
                put(wp, 0, f[4]), put(wp, 1, f[7]), put(wp, 2, f[8])
            f4, f7 = [f[4][1], down(f[4][0])], [down(f[7][0]), down(f[7][1])]
            f = [a0, a1, a2, a3, f4, a5, a6, f7, f[8]]
            F = Fn
            if hi and not lo:
                f[4], f[7], f[8] = mid(wp, 0), mid(wp, 1), mid(wp, 2)
            if it >= 2 * s:
                f, F = collide(s + 1, yn, f, F)
        p0, p1 = p1, p0
        y += 1


def emulate(S, fp64, nx, ny, H, glo=False, ghi=False):
    cols, first = 2 * (32 - S), S % 4
    stored = {}
    nstrips = (nx + cols - 1) // cols
    for item in range(nstrips * ((ny + H - 1) // H)):
        strip, ya = item % nstrips, item // nstrips * H
        march(S, fp64, nx, ny, strip * cols + first, min(cols, nx - strip * cols), ya, min(H, ny - ya), glo, ghi, stored)
    assert len(stored) == S * nx * ny and set(stored.values()) == {1}


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("S", [2, 4])
@pytest.mark.parametrize("nx,ny,H", [(4, 3, 1), (8, 4, 4), (52, 9, 3), (56, 7, 7), (60, 12, 5), (64, 5, 2), (112, 6, 6),
                                     (116, 8, 4), (124, 11, 1), (180, 6, 3)])
def test_strips(S, fp64, nx, ny, H):
    emulate(S, fp64, nx, ny, H)


@pytest.mark.parametrize("glo,ghi", [(True, False), (False, True), (True, True)])
def test_slab_ghost_rows(glo, ghi):
    emulate(2, False, 64, 9, 4, glo, ghi)
    emulate(2, True, 12, 5, 5, glo, ghi)


@pytest.mark.parametrize("waves", [1, 2, 4, 9])
@pytest.mark.parametrize("nx,ny,cols", [(4096, 2048, 60), (512, 256, 56), (200, 37, 60), (4, 3, 56), (60, 1 << 20, 60)])
def test_chunk_heights(waves, nx, ny, cols):
    """wave_grid: chunks of at least a row that cover the rows, at most the
    resident warps times the waves (or one per strip)"""
    occ, nsm, nw = 3, 148, 4
    nstrips = (nx + cols - 1) // cols
    chunks = min(ny, max(1, waves * occ * nsm * nw // nstrips))
    H = (ny + chunks - 1) // chunks
    n = (ny + H - 1) // H
    assert H >= 1 and n * H >= ny > (n - 1) * H and n <= chunks and nstrips * n < 1 << 31
