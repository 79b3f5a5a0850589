"""The mixed form's inversion, field by field, against the FP64 oracle.

Bound for every field and filtered spectrum, of its largest value: FP32 rounding
(6e-8) of about 14 operations a value (two transforms, right-hand sides,
recurrences), amplified by the solves, with ten times that as room: 3e-5.  (The
solves amplify the rounding of the longest waves of a flat box far more, but
these are a handful of modes among thousands.)
Needs a CUDA device."""
import math

import numpy as np
import pytest

from helpers import rel

pytestmark = pytest.mark.gpu
TWO_PI = 2 * math.pi


@pytest.mark.parametrize("shape", [(6, 4, 9), (36, 32, 7), (64, 60, 9), (72, 60, 20), (160, 64, 12), (160, 160, 6),
                                   (96, 96, 90), (72, 64, 180), (4, 4, 2500)])
def test_fields_of_the_mixed_inversion(shape):
    import pmpic_b200 as pm
    from oracle import Oracle
    nx, ny, nz = shape
    lz = math.pi * nz / max(nx, ny)
    rng = np.random.default_rng(nx + 10 * nz)
    f = {k: rng.standard_normal((nz + 1, ny, nx)) for k in ("p", "q", "r")}
    o = Oracle(nx, ny, nz, TWO_PI, TWO_PI, lz, max_parcels=8)
    g = pm.Context(nx, ny, nz, TWO_PI, TWO_PI, lz, max_parcels=8, precision="mixed")
    for k in f:
        o.set_grid(k, f[k])
        g.set_grid(k, f[k])
    o.vort2vel_grids()
    g.vort2vel_grids()
    for k in ("p", "q", "r", "u", "v", "w"):
        assert rel(g.grid(k), o.grid(k)) < 3e-5, k
    for k in ("u_s", "v_s", "w_s"):
        assert rel(g.spec(k), o.spec(k)) < 3e-5, k
    g.close()
    o.close()
