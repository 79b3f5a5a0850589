"""vort2vel's inversion with each tile width and CTA size that its rule picks, against the oracle.

The shapes lie on either side of the rule's lines: as many tiles as fit the
device at once with 8, 16 and 32 columns, more tiles than that, and columns
long enough that three CTAs no longer share an SM.  Bounds as for the other
shapes: FP64 differs by rounding (1e-16 times a condition number well below
1e4), the mixed form by FP32 rounding of fields and tables.
Needs a CUDA device."""
import math

import numpy as np
import pytest

from helpers import rel

pytestmark = pytest.mark.gpu
TWO_PI = 2 * math.pi


@pytest.mark.parametrize("shape", [(36, 32, 7), (64, 60, 9), (72, 60, 20), (160, 64, 12), (160, 160, 6), (96, 96, 90),
                                   (72, 64, 180)])
def test_inversion_plans_vs_oracle(shape):
    import pmpic_b200 as pm
    from oracle import Oracle
    nx, ny, nz = shape
    lz = math.pi * nz / max(nx, ny)
    rng = np.random.default_rng(nx + 10 * nz)
    f = {k: rng.standard_normal((nz + 1, ny, nx)) for k in ("p", "q", "r")}
    o = Oracle(nx, ny, nz, TWO_PI, TWO_PI, lz, max_parcels=8)
    for k in f:
        o.set_grid(k, f[k])
    o.vort2vel_grids()
    for prec, bound in (("fp64", 1e-11), ("mixed", 1e-3)):
        g = pm.Context(nx, ny, nz, TWO_PI, TWO_PI, lz, max_parcels=8, precision=prec)
        for k in f:
            g.set_grid(k, f[k])
        g.vort2vel_grids()
        for k in ("p", "q", "r", "u", "v", "w"):
            assert rel(g.grid(k), o.grid(k)) < bound, (prec, k)
        for k in ("u_s", "v_s", "w_s"):
            assert rel(g.spec(k), o.spec(k)) < bound, (prec, k)
        g.close()
    o.close()
