"""grid2par of six grids on boxes that the packed copy's launch cannot hold.

A launch has at most 65,535 blocks in y and in z, which the packing gives to 16
levels and to a row each; boxes beyond either are read from the grids
themselves, with the same operations.  Needs a CUDA device."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TWO_PI = 2 * math.pi
GRIDS, PROPS = ["u", "v", "w", "dp", "dq", "dr"], ["dxdt", "dydt", "dzdt", "dpdt", "dqdt", "drdt"]


@pytest.mark.parametrize("shape,n", [((4, 65536, 3), 600000), ((4, 60000, 3), 600000), ((4, 4, 1048559), 8400000),
                                     ((4, 4, 1048560), 8400000)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_six_grids_as_one_by_one(shape, n, precision):
    import pmpic_b200 as pm
    nx, ny, nz = shape
    rng = np.random.default_rng(ny)
    c = pm.Context(nx, ny, nz, TWO_PI, TWO_PI, math.pi, max_parcels=n + 8, precision=precision)
    c.upload(x=rng.uniform(0, TWO_PI, n), y=rng.uniform(0, TWO_PI, n), z=rng.uniform(0, math.pi, n), vol=np.ones(n))
    for k in GRIDS:
        c.set_grid(k, rng.standard_normal((nz + 1, ny, nx)))
    for g, p in zip(GRIDS, PROPS):  # one grid is never packed
        c.grid2par_multi([g], [p])
    want = {p: c.get(p, n) for p in PROPS}
    for p in PROPS:
        c.set(p, np.zeros(n), n)
    c.grid2par_multi(GRIDS, PROPS)
    for p in PROPS:
        np.testing.assert_array_equal(c.get(p, n), want[p], err_msg=p)
    c.close()
