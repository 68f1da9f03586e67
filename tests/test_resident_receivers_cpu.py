"""Receivers per tile of a resident tiling: the counts by which a tiling is chosen are those of the
lists that it runs with, for evenly spread, one-sided and vertical arrays on tilings that divide the
mesh unevenly."""
import ctypes as C
import random

import numpy as np
import pytest

from mun_b200 import _lib


def _counts(npol, nelx, nelz, elements, ntx, ntz):
    base = np.ascontiguousarray(np.array(elements, dtype=np.int32).reshape(-1, 2) * npol)
    out = [(C.c_int32 * 4)(), (C.c_int32 * 4)()]
    _lib.check(_lib.load().sem_selftest_receivers(npol, nelx, nelz, len(base), base.ctypes.data, ntx, ntz, *out))
    return tuple(tuple(o) for o in out)


def _by_nodes(npol, nelx, nelz, elements, ntx, ntz):
    """The fullest tile's counts from the nodes themselves."""
    def tile(g, nel, n):
        return next(t for t in reversed(range(n)) if min(g // npol, nel - 1) >= -(-t * nel // n))
    rec, inj, quads, terms = {}, {}, {}, {}
    for r, (ex, ez) in enumerate(elements):
        own = tile(ex * npol, nelx, ntx), tile(ez * npol, nelz, ntz)
        rec.setdefault(own, set()).add(r)
        for j in range(npol + 1):
            for i in range(npol + 1):
                gx, gz = ex * npol + i, ez * npol + j
                t = tile(gx, nelx, ntx), tile(gz, nelz, ntz)
                inj.setdefault(t, set()).add(r)
                quads.setdefault(t, set()).add((gz, gx // npol))
                terms.setdefault(t, set()).add((gz, gx // npol, r))
    return tuple(max((len(v) for v in d.values()), default=0) for d in (rec, inj, quads, terms))


def test_one_sided_vertical_array():
    elements = [(9, 3 + i * 7 // 81) for i in range(81)]
    counted, listed = _counts(5, 56, 31, elements, 2, 4)
    assert counted == listed == _by_nodes(5, 56, 31, elements, 2, 4)


@pytest.mark.parametrize("seed", range(12))
def test_counts_equal_the_lists(seed):
    rng = random.Random(seed)
    for _ in range(12):
        npol, nelx, nelz = rng.randint(1, 7), rng.randint(1, 40), rng.randint(1, 25)
        ntx, ntz = rng.randint(1, min(nelx, 9)), rng.randint(1, min(nelz, 9))
        x0, z0 = rng.randrange(nelx), rng.randrange(nelz)
        x1, z1 = rng.choice([x0, nelx - 1]), rng.choice([z0, nelz - 1])
        elements = [(rng.randint(x0, x1), rng.randint(z0, z1)) for _ in range(rng.choice([0, 1, 5, 40]))]
        counted, listed = _counts(npol, nelx, nelz, elements, ntx, ntz)
        assert counted == listed == _by_nodes(npol, nelx, nelz, elements, ntx, ntz)
