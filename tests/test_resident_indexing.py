"""Index audit of the resident kernels' tiles and neighbour exchange, on the CPU: every word a
tile waits for is sent exactly once, by the tile that owns the node, to the place it is read
from; every owned node is advanced by exactly one thread; every access lies inside its array."""
import pytest


def pitch(lpe, v):
    return (v + 7) // 16 * 16 + 8 if lpe == 2 else 4 * ((v + 3) // 4 | 1)


class Layout:
    """The fields of ResLay that index arithmetic uses."""

    def __init__(self, N, lpe, exm, ezm, ezl):
        self.N, self.Rm, self.Cm, self.qx = N, ezm * N + 1, exm * N + 1, exm + 1
        self.Wp = pitch(lpe, (0 if N == 4 else 4) + N + (exm + 1) * N)
        self.Cp = pitch(lpe, (exm + 1) * N)
        self.rows = max(ezm, ezl + 1) * N
        self.H = N + self.rows + 1
        self.t = self.Rm * N
        self.r = self.t + self.Cm * N
        self.b = self.r + self.Rm
        self.c = self.b + self.Cm
        self.words = self.c + 1


class Tile:
    def __init__(self, N, nelx, nelz, ntx, ntz, t):
        tx, tz = t % ntx, t // ntx
        ex0, ex1 = -(-tx * nelx // ntx), -(-(tx + 1) * nelx // ntx)
        ez0, ez1 = -(-tz * nelz // ntz), -(-(tz + 1) * nelz // ntz)
        self.EX, self.EZ = ex1 - ex0, ez1 - ez0
        self.hl, self.hr, self.ht, self.hb = ex0 > 0, ex1 < nelx, ez0 > 0, ez1 < nelz
        self.gx0, self.gz0 = ex0 * N, ez0 * N
        self.C, self.R = self.EX * N + (not self.hr), self.EZ * N + (not self.hb)
        self.X0 = (self.gx0 - N) & ~3
        self.off = self.gx0 - N - self.X0


def polls(T, L):
    """(word, region row, region column) in the kernel's order."""
    N = L.N
    for w in range(T.R * N if T.hl else 0):
        yield w, N + w // N, T.off + w % N
    for w in range(T.C * N if T.ht else 0):
        yield L.t + (w // T.C) * L.Cm + w % T.C, w // T.C, T.off + N + w % T.C
    for w in range(T.R if T.hr else 0):
        yield L.r + w, N + w, T.off + N + T.EX * N
    for w in range(T.C if T.hb else 0):
        yield L.b + w, N + T.R, T.off + N + w
    if T.hr and T.hb:
        yield L.c, N + T.R, T.off + N + T.EX * N


def sends(T, L, t, ntx):
    """(receiver, word, row, column) of every node a tile sends."""
    N = L.N
    QX = T.EX + (not T.hr)
    for r in range(T.R):
        for e in range(QX):
            lanes = range(N) if e < T.EX else range(1)
            if T.hr and e == T.EX - 1:
                for i in range(N):
                    yield t + 1, r * N + i, r, e * N + i
            if T.hl and e == 0:
                yield t - 1, L.r + r, r, 0
            if T.hb and r >= T.R - N:
                for i in lanes:
                    yield t + ntx, L.t + (r - (T.R - N)) * L.Cm + e * N + i, r, e * N + i
            if T.ht and r == 0:
                for i in lanes:
                    yield t - ntx, L.b + e * N + i, r, e * N + i
                if T.hl and e == 0:
                    yield t - ntx - 1, L.c, r, 0


@pytest.mark.parametrize("N,nelx,nelz,ntx,ntz,lpe", [
    (1, 7, 5, 3, 2, 1), (2, 9, 4, 4, 4, 1), (3, 11, 7, 3, 3, 1), (4, 10, 6, 10, 6, 1), (4, 10, 6, 10, 6, 2),
    (4, 13, 9, 4, 3, 1), (4, 13, 9, 4, 3, 2), (4, 5, 3, 1, 1, 2), (4, 14, 3, 1, 1, 2), (4, 30, 3, 1, 1, 1),
    (4, 8, 8, 1, 5, 1), (4, 8, 8, 1, 5, 2), (5, 7, 9, 3, 2, 1), (6, 5, 5, 2, 3, 1), (7, 4, 4, 3, 2, 1)])
def test_exchange_and_bounds(N, nelx, nelz, ntx, ntz, lpe):
    exm, ezm = -(-nelx // ntx), -(-nelz // ntz)
    L = Layout(N, lpe, exm, ezm, nelz // ntz)
    tiles = [Tile(N, nelx, nelz, ntx, ntz, t) for t in range(ntx * ntz)]
    assert sum(T.R * T.C for T in tiles) == (nelx * N + 1) * (nelz * N + 1)
    sent = {}
    for t, T in enumerate(tiles):
        assert 1 <= T.EX <= exm and 1 <= T.EZ <= ezm and T.X0 % 4 == 0 and 0 <= T.off <= 3
        for to, word, r, c in sends(T, L, t, ntx):
            assert 0 <= to < len(tiles) and 0 <= word < L.words
            assert (to, word) not in sent
            # a packed word's fields: place, offset of the receiver's tile, region index
            dx, dz = to % ntx - t % ntx, to // ntx - t // ntx
            assert word < 4096 and abs(dx) <= 1 and abs(dz) <= 1 and to == t + dx + dz * ntx
            assert (N + r) * L.Wp + T.off + N + c < min(65536, L.Wp * L.H)
            sent[to, word] = (T.gx0 + c, T.gz0 + r)
    wanted = set()
    for t, T in enumerate(tiles):
        for word, row, col in polls(T, L):
            assert 0 <= row < L.H and 0 <= col < L.Wp
            # the node of that place in the tile's region is the node that was sent there
            assert sent[t, word] == (T.X0 + col, T.gz0 - N + row)
            wanted.add((t, word))
    assert wanted == set(sent)
    # lanes: every owned node is advanced by exactly one thread; reads stay inside the arrays
    sw = 4
    nj = N // lpe
    while sw < (exm + 2) * lpe:
        sw *= 2
    for ezc in (1, 2, 3):
        for T in tiles:
            seen = set()
            ez1 = T.EZ + (not T.hb)
            for ch in range(-(-max(ezm, nelz // ntz + 1) // ezc)):
                lo, hi = ch * ezc, min(ez1, ch * ezc + ezc)
                first = min(lo, ez1 - 1)
                assert N + first * N < L.H and (not (lo < hi and (lo > 0 or T.ht)) or first * N >= 0)
                for sl in range(sw):
                    el, h = sl // lpe, sl % lpe
                    ec = min(el - 1, T.EX)
                    full = 1 <= el <= T.EX
                    owner = full or (el == T.EX + 1 and not T.hr)
                    col = T.off + N + ec * N
                    assert col >= 0 and col + N + (N & 1) <= L.Wp
                    assert not full or sl + lpe < sw  # the next lane holds the nodes on the right
                    for er in range(lo, lo + ezc):
                        e_ = min(er, ez1 - 1)
                        assert N + e_ * N + N < L.H and e_ * N + N <= L.rows
                        assert not owner or (ec + 1) * N <= L.Cp and ec < L.qx
                        if owner and er < hi:
                            for j in range(nj):
                                r = e_ * N + h * nj + j
                                if e_ == T.EZ and r > T.EZ * N:
                                    continue
                                for i in range(N if full else 1):
                                    assert (r, ec * N + i) not in seen
                                    seen.add((r, ec * N + i))
                                    # the warp that sends a node's exchange words is the one that advances it
                                    assert ch * sw + (ec + 1) * lpe + (r % N) // nj == ch * sw + sl
            assert seen == {(r, c) for r in range(T.R) for c in range(T.C)}
            # receivers' elements, the corner node included, lie inside the region
            assert N + (T.EZ - 1) * N + N < L.H and T.off + N + (T.EX - 1) * N + N < L.Wp
