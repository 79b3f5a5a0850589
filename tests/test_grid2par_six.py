"""grid2par of six grids at once against the same six in two calls of three.

Six grids are gathered from a packed copy when there are enough parcels (at
least 65,536, and one to two grid points), three from the grids themselves;
the operations are the same, so the values are equal bit for bit, on either
side of the limit and on shapes whose sides leave remainders in the packing's
32 x 16 tiles.  Needs a CUDA device."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TWO_PI = 2 * math.pi
GRIDS = ["u", "v", "w", "dp", "dq", "dr"]
SIX = ["dxdt", "dydt", "dzdt", "dpdt", "dqdt", "drdt"]


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("shape,n", [((36, 30, 17), 65535), ((36, 30, 17), 65536), ((4, 6, 3), 70001),
                                     ((50, 64, 47), 76799), ((50, 64, 47), 76800), ((64, 80, 33), 100000)])
def test_six_grids_equal_three_and_three(shape, n, prec):
    import pmpic_b200 as pm
    nx, ny, nz = shape
    rng = np.random.default_rng(n)
    lo = 1e-9  # a position on the upper wall belongs to no cell
    pos = {k: rng.uniform(0, length * (1 - lo), n) for k, length in zip("xyz", (TWO_PI, TWO_PI, math.pi))}
    zero = np.zeros(n)
    c = pm.Context(nx, ny, nz, TWO_PI, TWO_PI, math.pi, max_parcels=n, precision=prec)
    c.upload(**pos, vol=np.ones(n), **{k: zero for k in ("p", "q", "r", "b", "h", "stretch", "tag")})
    for k in GRIDS:
        c.set_grid(k, rng.standard_normal((nz + 1, ny, nx)))
    c.grid2par_multi(GRIDS, SIX)
    six = [c.get(k, n) for k in SIX]
    c.grid2par_multi(GRIDS[:3], SIX[:3])
    c.grid2par_multi(GRIDS[3:], SIX[3:])
    for k, v in zip(SIX, six):
        assert np.abs(v).max() > 0
        assert np.array_equal(c.get(k, n), v), k
    c.close()
