"""The transforms and the two spectral components over the row lengths.

Every even length with the prime factors 2, 3 and 5 up to 256 is either a
product of two register radices (2 .. 16, the four-step kernels) or, with
those above 256, a Stockham row; these shapes take each radix in each pass,
columns that do not fill a CTA of 16, and one direction of each kind.
Needs a CUDA device."""
import math

import numpy as np
import pytest

from helpers import rel

pytestmark = pytest.mark.gpu
TWO_PI = 2 * math.pi
SHAPES = [(4, 4, 3), (4, 36, 3), (6, 10, 5), (8, 6, 4), (12, 18, 4), (18, 12, 4), (20, 24, 5), (24, 20, 3),
          (30, 54, 3), (36, 30, 4), (40, 50, 3), (48, 96, 5), (60, 40, 3), (72, 90, 3), (80, 108, 3), (90, 60, 3),
          (96, 48, 5), (100, 72, 3), (108, 80, 3), (120, 100, 3), (144, 120, 3), (150, 8, 4), (160, 150, 3),
          (180, 16, 3), (192, 180, 3), (240, 192, 3), (16, 240, 3), (128, 144, 4), (10, 256, 3), (256, 16, 3),
          (162, 12, 3), (12, 200, 3), (320, 8, 3), (8, 320, 3), (216, 250, 3)]


@pytest.fixture(scope="module")
def pm():
    import pmpic_b200
    return pmpic_b200


@pytest.mark.parametrize("shape", SHAPES)
def test_transforms_vs_numpy_and_oracle(pm, shape):
    from oracle import Oracle
    nx, ny, nz = shape
    g = pm.Context(nx, ny, nz, TWO_PI, TWO_PI, math.pi, max_parcels=8)
    o = Oracle(nx, ny, nz, TWO_PI, TWO_PI, math.pi, max_parcels=8)
    rng = np.random.default_rng(nx * 1000 + ny)
    f = rng.standard_normal((nz + 1, ny, nx))
    s = g.fft_forward(f)
    assert rel(s, o.fft_forward(f)) < 1e-13
    assert rel(g.fft_backward(s), f) < 1e-13
    s = rng.standard_normal(s.shape)
    assert rel(g.fft_backward(s), o.fft_backward(s)) < 1e-13
    g.close()
    o.close()


@pytest.mark.parametrize("shape", SHAPES)
def test_components_vs_oracle(pm, shape):
    """vort2vel and vorticity_tendency of random parcels: FP64 to the rounding of the transforms and the
    par2grid sums (their derivatives amplified by the largest wavenumber over the mean one), FP32 likewise."""
    from oracle import Oracle
    nx, ny, nz = shape
    rng = np.random.default_rng(nx + 7 * ny)
    n = 4 * nx * ny * nz
    p = {"x": rng.uniform(0, TWO_PI, n), "y": rng.uniform(0, TWO_PI, n), "z": rng.uniform(0, math.pi, n),
         "vol": rng.uniform(0.5, 1.5, n) * TWO_PI * TWO_PI * math.pi / n}
    for k in ("p", "q", "r", "b"):
        p[k] = rng.standard_normal(n)
    p["h"] = 0.5 * rng.uniform(size=n)
    o = Oracle(nx, ny, nz, TWO_PI, TWO_PI, math.pi, max_parcels=n + 8)
    o.set_parcels(**p)
    o.vort2vel()
    o.vorticity_tendency()
    for prec, bound in (("fp64", 1e-11), ("mixed", 1e-3)):
        g = pm.Context(nx, ny, nz, TWO_PI, TWO_PI, math.pi, max_parcels=n + 8, precision=prec)
        g.upload(**p)
        g.vort2vel()
        g.vorticity_tendency()
        for k in ("u", "v", "w", "p", "q", "r", "b", "dp", "dq", "dr"):
            assert rel(g.grid(k), o.grid(k)) < bound, (prec, k)
        for k in ("u_s", "v_s", "w_s"):
            assert rel(g.spec(k), o.spec(k)) < bound, (prec, k)
        g.close()
    o.close()
