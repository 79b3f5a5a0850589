"""The order of the cell index on unevenly filled cells: slots in cell order and,
within a cell, ascending, whichever way a cell's entries are sorted.

Needs a CUDA device."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TWO_PI = 2 * math.pi


def index_order(shape, counts, precision, seed):
    """Cell c holds counts[c % len(counts)] parcels, slots in random order: the tags after renumbering, and
    as a stable sort of the cells gives them."""
    import pmpic_b200 as pm
    nx, ny, nz = shape
    rng = np.random.default_rng(seed)
    cell = rng.permutation(np.repeat(np.arange(nx * ny * nz), np.resize(counts, nx * ny * nz)))
    n = len(cell)
    ijk = (cell // (ny * nz), cell // nz % ny, cell % nz)
    d = (TWO_PI / nx, TWO_PI / ny, math.pi / nz)
    p = {k: d[v] * (ijk[v] + rng.uniform(0.01, 0.99, n)) for v, k in enumerate("xyz")}
    p["vol"], p["tag"] = np.ones(n), np.arange(n, dtype=np.float64)
    c = pm.Context(nx, ny, nz, TWO_PI, TWO_PI, math.pi, max_parcels=n + 8, precision=precision)
    c.upload(**p)
    c.sort_parcels()
    got = c.get("tag")
    c.close()
    return got, np.argsort(cell, kind="stable").astype(np.float64)


# (a warp's 32 cells hold the pattern once): either side of 16 entries, of a fullest cell of 56, and of
# three times the ranking steps against the square of the fullest cell
@pytest.mark.parametrize("counts", [[8] * 32, [16] * 31 + [56], [17] * 31 + [57], [27, 20, 35, 31], [56] * 32, [57] + [8] * 31,
                                    [17] * 6 + [2] * 25 + [56], [48] * 8 + [8] * 24, [48] * 7 + [8] * 25, [0] * 31 + [17]])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_which_cells_are_ranked(counts, precision):
    got, want = index_order((8, 6, 16), counts, precision, 7)
    np.testing.assert_array_equal(got, want)


# cells that a warp and that the whole CTA ranks, CTAs whose 256 cells hold more than the 8192 entries that
# are staged at a time, cells of just 8192 and more, and all of these beside ordinary and empty ones
@pytest.mark.parametrize("counts", [[33], [64], [256, 257], [513, 0, 8], [700, 3], [8191, 1, 8], [8192, 8], [8193, 17, 64],
                                    [9000, 0, 0, 40, 40], [30] * 31 + [8192], [2000, 6000, 192, 1]])
@pytest.mark.parametrize("shape", [(4, 4, 3), (8, 6, 11)])
def test_staged_in_passes(counts, shape):
    if sum(counts) / len(counts) * np.prod(shape) > 2e6:
        counts = counts + [8] * 30
    got, want = index_order(shape, counts, "fp64", 9)
    np.testing.assert_array_equal(got, want)
