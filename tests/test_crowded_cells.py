"""The cell index, par2grid and the mixing grids on unevenly filled cells.

A cell's slots are sorted by one thread up to 16 of them, ranked by its warp up
to 512, and sorted in place when 256 neighbouring cells hold more than the
8192 that are staged; slots in random order put cells on both sides of each
line, with empty cells and uneven columns beside them.  Needs a CUDA device."""
import math

import numpy as np
import pytest

from helpers import rel

pytestmark = pytest.mark.gpu
TWO_PI = 2 * math.pi


@pytest.fixture(scope="module")
def pm():
    import pmpic_b200
    return pmpic_b200


def crowded(shape, counts, seed):
    """Parcels at random places of their cells, cell c holding counts[c % len(counts)] of them, in random slot order."""
    nx, ny, nz = shape
    rng = np.random.default_rng(seed)
    cell = np.repeat(np.arange(nx * ny * nz), np.resize(counts, nx * ny * nz))
    cell = rng.permutation(cell)
    n = len(cell)
    d = (TWO_PI / nx, TWO_PI / ny, math.pi / nz)
    ijk = (cell // (ny * nz), cell // nz % ny, cell % nz)
    p = {k: d[v] * (ijk[v] + rng.uniform(0.01, 0.99, n)) for v, k in enumerate("xyz")}
    p["vol"] = rng.uniform(0.5, 1.5, n) * d[0] * d[1] * d[2] / 8
    for k in ("p", "q", "r", "b", "h"):
        p[k] = rng.standard_normal(n)
    p["tag"] = np.arange(n, dtype=np.float64)
    p["stretch"] = np.zeros(n)
    return p


COUNTS = [[15], [16, 17], [17], [32, 33], [64], [128, 0, 129], [300, 0, 1], [512, 0, 0], [513, 1, 0, 0],
          [64, 8, 8, 64], [4, 4, 4, 4, 4, 4, 4, 100]]


@pytest.mark.parametrize("shape", [(8, 6, 5), (10, 4, 18)])
@pytest.mark.parametrize("counts", COUNTS)
def test_par2grid_crowded_cells_vs_oracle(pm, shape, counts):
    from oracle import Oracle
    p = crowded(shape, counts, 3 + len(counts))
    cap = len(p["x"]) + 16
    o = Oracle(*shape, TWO_PI, TWO_PI, math.pi, max_parcels=cap)
    o.set_parcels(**p)
    cells = o.cache_weights()
    f = ["p", "q", "r", "b"]
    for k in f:
        o.par2grid(k, k)
    # FP64: sums of at most 8 * 513 terms in another order; FP32: their rounding (and the offsets')
    for prec, bound in (("fp64", 1e-12), ("mixed", 1e-4)):
        c = pm.Context(*shape, TWO_PI, TWO_PI, math.pi, max_parcels=cap, precision=prec)
        c.upload(**p)
        np.testing.assert_array_equal(c.cell_ids(), cells)
        for seg in (1, 3, 64):  # a column's sums do not depend on the segment that holds it
            pm.lib().pmpic_set_p2g_segment(c._h, seg)
            c.par2grid_multi(f, f)  # (bins and sorts afresh)
            got = {k: c.grid(k) for k in f}
            if seg == 1:
                first = got
            for k in f:
                assert rel(got[k], o.grid(k)) < bound, (prec, seg, k)
                np.testing.assert_array_equal(got[k], first[k])
        # the index itself: after renumbering, slots are in cell order and, within a cell, in the old slot order
        c.sort_parcels()
        order = np.argsort((cells // shape[0] % shape[1] + cells % shape[0] * shape[1]) * shape[2]
                           + cells // (shape[0] * shape[1]), kind="stable")
        np.testing.assert_array_equal(c.get("tag"), p["tag"][order])
        c.close()
    o.close()


@pytest.mark.parametrize("counts", [[17], [64, 2, 8], [129, 0, 3]])
def test_mixing_crowded_cells_vs_oracle(pm, counts):
    from oracle import Oracle
    shape = (8, 6, 6)
    p = crowded(shape, counts, 11)
    n = len(p["x"])
    vmin = (TWO_PI / 8) * (TWO_PI / 6) * (math.pi / 6) / 216
    p["vol"][np.random.default_rng(5).uniform(size=n) < 0.1] = 0.5 * vmin
    cap = 2 * n + 1024
    c = pm.Context(*shape, TWO_PI, TWO_PI, math.pi, max_parcels=cap)
    o = Oracle(*shape, TWO_PI, TWO_PI, math.pi, max_parcels=cap)
    c.upload(**p)
    o.set_parcels(**p)
    for _ in range(4):  # mixing acts on the fourth call
        c.parcel_mixing()
        o.parcel_mixing()
    assert c.n == o.n
    ci, oi = c.info(), o.info()
    assert (ci.n_removed, ci.n_added) == (oi.n_removed, oi.n_added) and ci.n_removed > 0
    np.testing.assert_array_equal(c.get("tag"), o.get("tag"))
    for k in ("x", "y", "z", "vol", "b", "h", "p", "q", "r"):
        assert rel(c.get(k), o.get(k)) < 1e-11, k
    c.close()
    o.close()
