"""Context creation: the tables that its kernels derive on the device.

Needs a CUDA device."""
import math

import numpy as np
import pytest

from helpers import rel

pytestmark = pytest.mark.gpu
TWO_PI = 2 * math.pi


@pytest.mark.parametrize("shape", [(64, 64, 64), (48, 40, 150)])
def test_fresh_contexts_have_the_same_tables(shape):
    """Contexts made one after the other, each used at once: the FP64 inversion's factors are derived on the
    device from copies of host tables, so a creation that did not wait for them would differ from the others
    and from the oracle.  Same inputs, fixed summation orders: equal bits; 1e-11 as for other shapes (FP64
    rounding, 1e-16, times a condition number well below 1e4)."""
    import pmpic_b200 as pm
    from oracle import Oracle
    nx, ny, nz = shape
    lz = math.pi * nz / max(nx, ny)
    rng = np.random.default_rng(nz)
    f = {k: rng.standard_normal((nz + 1, ny, nx)) for k in ("p", "q", "r")}
    o = Oracle(nx, ny, nz, TWO_PI, TWO_PI, lz, max_parcels=8)
    for k in f:
        o.set_grid(k, f[k])
    o.vort2vel_grids()
    want = None
    for _ in range(6):
        g = pm.Context(nx, ny, nz, TWO_PI, TWO_PI, lz, max_parcels=8)
        for k in f:
            g.set_grid(k, f[k])
        g.vort2vel_grids()
        got = {k: g.grid(k) for k in ("p", "q", "r", "u", "v", "w")}
        g.close()
        for k in got:
            assert rel(got[k], o.grid(k)) < 1e-11, k
            if want is not None:
                np.testing.assert_array_equal(got[k], want[k], err_msg=k)
        want = got
    o.close()


@pytest.mark.parametrize("nz", [1022, 1023, 1024, 2048, 7300])
def test_mixed_form_of_any_depth(nz):
    """The mixed form's mean flow passes through shared memory 1024 levels at a time; a context of more levels
    than shared memory would hold at once (7264) is made and inverts.  Bound: FP32 rounding (6e-8) of about
    14 operations a value (transforms of length 4, right-hand sides, recurrences), amplified by at most 4
    (off-diagonals 0.38 of the diagonal), with ten times that as room."""
    import pmpic_b200 as pm
    from oracle import Oracle
    lz = math.pi * nz / 4
    rng = np.random.default_rng(nz)
    f = {k: rng.standard_normal((nz + 1, 4, 4)) for k in ("p", "q", "r")}
    o = Oracle(4, 4, nz, TWO_PI, TWO_PI, lz, max_parcels=8)
    g = pm.Context(4, 4, nz, TWO_PI, TWO_PI, lz, max_parcels=8, precision="mixed")
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
