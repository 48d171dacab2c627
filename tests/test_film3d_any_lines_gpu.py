"""Film_3D sweeps on lines of any length (4 to 32 lanes with K or K - 1 rows
each, the shapes' first and last lengths) in both precisions against the FP64
oracle, and the serial recurrence of systems that are not diagonally dominant
with its pivot checks."""
import numpy as np
import pytest

from adscf_gb300 import FILM_3D, FP64, SPLIT, Context
from adscf_gb300._lib import AdscfError
from oracle import film as of

pytestmark = pytest.mark.gpu

SHAPES = [(9, 9, 8), (20, 35, 24), (21, 13, 20), (40, 41, 39), (17, 80, 40), (81, 10, 79), (12, 160, 9),
          (9, 11, 159), (33, 27, 80), (8, 9, 12), (16, 161, 10)]      # the last two: one thread per line


def film(grid, ns, prec):
    gx, gy, gz = grid
    depth = 0.08 * gz
    z = np.arange(gz + 1) / gz
    zr = depth * (z + 0.05 * np.sin(2 * np.pi * z) / (2 * np.pi))
    dz = of.mesh_from_zr(zr)
    return dict(grid=grid, size=(0.11 * gx, 0.09 * gy, depth), dz=dz, dss=of.contour_steps(ns, ds_scheme=1),
                n_a=ns // 2, block_length=(0.5, 0.5), chi=15.0, kappa=25.0, int_scheme=1, int_span=0, ensemble=2,
                mu=0.3, precision=prec)


# FP64: rounding times the matrices' O(ds / h^2) ~ 10 over ten steps; split:
# FP32 rounding of the increments, 6e-8 a step, over ten steps and two orders
# of margin for the thin films' decay
@pytest.mark.parametrize("prec,tol", [(FP64, 1e-12), (SPLIT, 2e-5)])
@pytest.mark.parametrize("grid", SHAPES)
def test_chains_vs_oracle(rng, grid, prec, tol):
    kw = film(grid, 10, prec)
    gx, gy, gz = grid
    w = rng.standard_normal((2, gz + 1, gy, gx))
    w[:, 0] = w[:, -1] = 0.0
    dx, dy = kw["size"][0] / gx, kw["size"][1] / gy
    step = lambda p, f, ds: of.adi_step_3d(p, f, kw["dz"], dx, dy, ds)  # noqa: E731
    ref = of.film_propagate_diblock(w, kw["dz"], kw["dss"], kw["n_a"], step, dx=dx, dy=dy, int_scheme=1, span="full",
                                    ensemble=2, mu=0.3, sizes=kw["size"])
    if ref["Qsum"] <= 0:
        pytest.skip("ten steps leave this film's Q negative")
    with Context(FILM_3D, **kw) as c:
        dens, res = c.propagate_diblock(w)
    assert abs(res.Qsum / ref["Qsum"] - 1.0) < tol
    assert np.max(np.abs(dens - ref["density"])) < 5 * tol * np.max(np.abs(ref["density"]))


@pytest.mark.parametrize("prec,tol", [(FP64, 1e-12), (SPLIT, 1e-4)])
def test_systems_that_are_not_dominant(rng, prec, tol):
    grid = (11, 20, 12)
    kw = film(grid, 10, prec)
    ds, h = 0.1, kw["size"]
    q = 1.0 + 0.1 * rng.standard_normal((13, 20, 11))
    w = rng.standard_normal(q.shape)
    w[4, 3, 2] = w[5, 3, 2] = w[7, 19, 10] = -2.5 / ds
    with Context(FILM_3D, **kw) as c:
        got = c.propagate_step(q, w, ds)
    want = of.adi_step_3d(q, w, kw["dz"], h[0] / 11, h[1] / 20, ds)
    # walls keep the reference's values; the bound scales with the solution
    assert np.max(np.abs(got - want)[1:-1]) < tol * np.max(np.abs(want))


@pytest.mark.parametrize("plane,w0", [(1, -16.0), (2, -15.0)])
def test_zero_pivots(plane, w0):
    """h = 0.5, ds = 0.25 in z: a = c = -1/2 and diagonals 2, so -16 at plane 1
    or -15 at plane 2 of one line is a zero pivot of the recurrence."""
    gz = 12
    dz = np.r_[0.0, np.full(gz, 0.5)]
    w = np.zeros((gz + 1, 10, 9))
    w[plane, 4, 5] = w0
    with Context(FILM_3D, grid=(9, 10, gz), size=(4.5, 5.0, 6.0), dz=dz, ds=0.25, block_length=(0.5, 0.5),
                 precision=FP64) as c:
        with pytest.raises(AdscfError) as e:
            c.propagate_step(np.ones(w.shape), w, 0.25)
        assert e.value.code == 3
