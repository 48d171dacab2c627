"""Film_3D sweeps at the limits of the lines they take (9 and 160 rows, planes that
fill a block's shared memory) and just past them (8 and 161 rows, FP64 planes that do
not fit), where a thread solves a line, in films deep enough that Q stays positive."""
import numpy as np
import pytest

from adscf_gb300 import FILM_3D, FP64, SPLIT, Context, _lib
from oracle import film as of

pytestmark = pytest.mark.gpu

NS = 10
# kernels of a propagation: 1 + factors + 2 a step on lines of any length, 1 + 3 a step with a thread per line
ANY, THREAD = 2 + 2 * NS, 1 + 3 * NS


def film(grid, prec):
    gx, gy, gz = grid
    depth = 4.0 + 0.08 * gz
    z = np.arange(gz + 1) / gz
    dz = of.mesh_from_zr(depth * (z + 0.05 * np.sin(2 * np.pi * z) / (2 * np.pi)))
    return dict(grid=grid, size=(0.11 * gx, 0.09 * gy, depth), dz=dz, dss=of.contour_steps(NS, ds_scheme=1), n_a=NS // 2,
                block_length=(0.5, 0.5), chi=15.0, kappa=25.0, int_scheme=1, int_span=0, ensemble=2, mu=0.3,
                precision=prec)


# FP64: rounding times the matrices' O(ds / h^2) ~ 10 over ten steps; split: FP32
# rounding of the increments, 6e-8 a step, times the same
@pytest.mark.parametrize("prec,tol", [(FP64, 1e-12), (SPLIT, 2e-5)])
@pytest.mark.parametrize("grid,launches", [((9, 9, 8), ANY), ((12, 160, 9), ANY), ((160, 9, 9), ANY), ((9, 10, 159), ANY),
                                           ((8, 9, 12), THREAD), ((9, 8, 12), THREAD), ((16, 161, 10), THREAD),
                                           ((9, 9, 7), THREAD), ((9, 9, 160), THREAD), ((112, 128, 9), ANY),
                                           ((114, 128, 9), THREAD), ((128, 128, 9), THREAD)])
def test_limits_vs_oracle(rng, grid, launches, prec, tol):
    kw = film(grid, prec)
    gx, gy, gz = grid
    w = rng.standard_normal((2, gz + 1, gy, gx))
    w[:, 0] = w[:, -1] = 0.0
    dx, dy = kw["size"][0] / gx, kw["size"][1] / gy
    step = lambda p, f, ds: of.adi_step_3d(p, f, kw["dz"], dx, dy, ds)  # noqa: E731
    ref = of.film_propagate_diblock(w, kw["dz"], kw["dss"], kw["n_a"], step, dx=dx, dy=dy, int_scheme=1, span="full",
                                    ensemble=2, mu=0.3, sizes=kw["size"])
    assert ref["Qsum"] > 0
    with Context(FILM_3D, **kw) as c:
        dens, res = c.propagate_diblock(w)
        got = c.lib.adscf_stage_launches(c.h, _lib.STAGE_PROPAGATE)
    if prec == FP64:                   # split contexts take what their tuner found faster
        assert got == launches
    assert abs(res.Qsum / ref["Qsum"] - 1.0) < tol
    assert np.max(np.abs(dens - ref["density"])) < 5 * tol * np.max(np.abs(ref["density"]))
