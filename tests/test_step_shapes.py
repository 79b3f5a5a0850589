"""Grid shapes and parcel counts at the edges of the kernels' tiles, against the oracle.

* vort2vel's inversion with every tile width and with more levels than shared
  memory holds (the columns then live in global memory);
* whole steps on ragged boxes (packed gather grids, haloswap, mixing);
* the cell scan either side of its one-launch limit, the haloswap's list
  either side of a compaction block (8192 parcels), and a split call in which
  nothing splits.
Needs a CUDA device."""
import math

import numpy as np
import pytest

from helpers import ALL, lattice_parcels, rel, rel_l2

pytestmark = pytest.mark.gpu
TWO_PI = 2 * math.pi


@pytest.fixture(scope="module")
def pm():
    import pmpic_b200
    return pmpic_b200


@pytest.mark.parametrize("shape", [(4, 4, 3), (6, 4, 9), (30, 6, 17), (36, 8, 40), (64, 64, 15), (80, 48, 31),
                                   (100, 96, 47), (16, 8, 160), (12, 6, 310), (8, 4, 700), (4, 6, 1300), (4, 4, 2500)])
def test_inversion_shapes_vs_oracle(pm, shape):
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


@pytest.mark.parametrize("shape", [(10, 6, 5), (36, 30, 17), (64, 8, 33), (18, 40, 16)])
def test_steps_on_ragged_boxes_vs_oracle(pm, shape):
    from oracle import Oracle
    nx, ny, nz = shape
    p = lattice_parcels(nx, ny, nz, TWO_PI, TWO_PI, math.pi)
    n = len(p["x"])
    rng = np.random.default_rng(n)
    d = (TWO_PI / nx, TWO_PI / ny, math.pi / nz)
    for k, h in zip("xyz", d):
        p[k] = p[k] + rng.uniform(-0.2, 0.2, n) * h
    p["vol"] = np.full(n, d[0] * d[1] * d[2] / 8)
    for k, ph in zip("pqr", (0.0, 0.7, 1.9)):
        p[k] = np.sin(p["x"] + ph) * np.cos(p["y"] - ph) * np.sin(p["z"])
    p["b"], p["h"] = np.cos(p["x"]) * 0.3, 0.2 + 0 * p["x"]
    p["tag"], p["stretch"] = np.arange(n, dtype=np.float64), np.zeros(n)
    cap = 2 * n
    o = Oracle(nx, ny, nz, TWO_PI, TWO_PI, math.pi, dtm=0.05, dtmax=0.05, max_parcels=cap)
    o.set_parcels(**p)
    ctx = {k: pm.Context(nx, ny, nz, TWO_PI, TWO_PI, math.pi, dtm=0.05, dtmax=0.05, max_parcels=cap, precision=k)
           for k in ("fp64", "mixed")}
    for g in ctx.values():
        g.upload(**p)
        g.step(3)
    for _ in range(3):
        o.step()
    for prec, bound in (("fp64", 1e-10), ("mixed", 1e-4)):
        g = ctx[prec]
        assert g.n == o.n
        np.testing.assert_array_equal(g.get("tag"), o.get("tag"))
        for k in ("u", "v", "w"):
            assert rel_l2(g.grid(k), o.grid(k)) < bound, (prec, k)
        g.close()
    o.close()


@pytest.mark.parametrize("shape", [(16, 16, 16), (16, 16, 17), (64, 64, 64), (64, 64, 65)])
def test_cell_scan_either_side_of_its_limits(pm, shape):
    from oracle import Oracle
    nx, ny, nz = shape
    n = 2 * nx * ny * nz
    rng = np.random.default_rng(nz)
    p = {"x": rng.uniform(0, TWO_PI, n), "y": rng.uniform(0, TWO_PI, n), "z": rng.uniform(0, math.pi, n),
         "vol": rng.uniform(0.5, 1.5, n), "b": rng.standard_normal(n)}
    o = Oracle(nx, ny, nz, TWO_PI, TWO_PI, math.pi, max_parcels=n)
    g = pm.Context(nx, ny, nz, TWO_PI, TWO_PI, math.pi, max_parcels=n)
    o.set_parcels(**p)
    g.upload(**p)
    np.testing.assert_array_equal(g.cell_ids(), o.cache_weights())
    o.par2grid("b", "b")
    g.par2grid("b", "b")
    assert rel(g.grid("b"), o.grid("b")) < 1e-12
    g.close()
    o.close()


@pytest.mark.parametrize("n", [1, 8191, 8192, 8193, 40000])
@pytest.mark.parametrize("share", [0.0, 0.02, 1.0])
def test_haloswap_lists_vs_oracle(pm, n, share):
    from oracle import Oracle
    rng = np.random.default_rng(n)
    out = rng.uniform(size=n) < share
    p = {k: rng.standard_normal(n) for k in ALL}
    for k, hi in (("x", TWO_PI), ("y", TWO_PI), ("z", math.pi)):
        p[k] = rng.uniform(0.0, hi, n)
    for k in "xy":
        p[k] = np.where(out, rng.uniform(-0.3, TWO_PI + 0.3, n), p[k])
    p["stretch"] = np.zeros(n)
    g = pm.Context(16, 16, 8, TWO_PI, TWO_PI, math.pi, max_parcels=n + 8)
    o = Oracle(16, 16, 8, TWO_PI, TWO_PI, math.pi, max_parcels=n + 8)
    for k in ALL:
        g.set(k, p[k], n)
    o.set_parcels(**p)
    g.set_count(n)
    o.set_count(n)
    g.parcel_haloswap()
    o.parcel_haloswap()
    assert g.info().n_migrated == o.info().n_migrated
    for k in ALL:
        np.testing.assert_array_equal(g.get(k), o.get(k), err_msg=k)
    # a split call that splits nothing leaves every parcel where it is
    g.set_counters([0, 0, 1, 3, 0])
    o.set_counters([0, 0, 1, 3, 0])
    g.set_dtm(0.0)
    o.set_dtm(0.0)
    g.parcel_splitting()
    o.parcel_splitting()
    assert (g.n, g.info().n_split, g.info().n_migrated) == (o.n, 0, 0)
    for k in ALL:
        np.testing.assert_array_equal(g.get(k), o.get(k), err_msg=k)
    g.close()
    o.close()
