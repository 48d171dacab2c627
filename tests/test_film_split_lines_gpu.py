"""Split-precision films on lines of several warps: many contour steps, so that
what a warp knows of its neighbours' edge rows may not drift from them, against
the same film in FP64."""
import numpy as np
import pytest

from adscf_gb300 import BRUSH, FILM_1D, FP64, SPLIT, Batch, Context
from oracle import film as of

pytestmark = pytest.mark.gpu


def film(rows, ns, prec):
    gz = rows - 1
    depth = 8.0
    dz = np.r_[0.0, np.full(gz, depth / gz)]
    dss = np.r_[0.0, np.full(ns, 1.0 / ns)]
    return dict(grid=(1, 1, gz), size=(1.0, 1.0, depth), dz=dz, dss=dss, n_a=ns // 2, block_length=(0.5, 0.5),
                int_scheme=1, int_span=1, ensemble=1, rho=1.0, precision=prec)


def fields(rng, rows):
    z = np.arange(rows) / (rows - 1)
    w = np.stack([s * 3.0 * np.cos(8 * np.pi * z) for s in (1, -1)]) + 0.05 * rng.standard_normal((2, rows))
    w[:, 0] = w[:, -1] = 0.0
    return w


# The split sweeps solve for increments, so a step's rounding is 6e-8 of the
# increment; over the contour the increments add up to some ten times q.
TOL = 6e-7


@pytest.mark.parametrize("rows", [257, 401, 801, 1501, 2001])
def test_many_steps_stay_at_fp32_rounding(rng, rows):
    w = fields(rng, rows).reshape(2, rows, 1, 1)
    got = []
    for prec in (FP64, SPLIT):
        with Context(FILM_1D, **film(rows, 1200, prec)) as c:
            got.append(c.propagate_diblock(w))
    (want, r64), (dens, r) = got
    assert abs(np.log(r.Qsum / r64.Qsum)) < TOL
    assert np.max(np.abs(dens - want)) < TOL * np.max(np.abs(want))


def test_batch_of_long_lines(rng):
    inst, w = [], []
    for rows in (300, 700, 1501):
        inst.append(dict(film(rows, 1200, SPLIT), geometry=FILM_1D, chi=15.0, kappa=25.0))
        w.append(fields(rng, rows).reshape(2, rows, 1, 1))
    with Batch(inst) as b:
        b.set_fields(w)
        b.scf_run(1)
        got = b.get_densities()
    for kw, wi, d in zip(inst, w, got):
        kw = dict(kw, precision=FP64)
        kw.pop("geometry")
        with Context(FILM_1D, **kw) as c:
            c.set_field(wi)
            c.scf_run(1)
            want = c.get_density()
        assert np.max(np.abs(d.ravel() - want)) < TOL * np.max(np.abs(want))


def test_brush(rng):
    rows, ns = 1001, 600
    kw = film(rows, ns, SPLIT)
    z = np.arange(rows) / (rows - 1)
    graft = np.exp(-0.5 * ((z - 0.05) / 0.01) ** 2)
    graft[0] = graft[-1] = 0.0
    w = 1.2 * np.exp(-3.0 * z) + 0.02 * rng.standard_normal(rows)
    w[0] = w[-1] = 0.0
    got = []
    for prec in (FP64, SPLIT):
        kw.update(precision=prec, graft=graft / of.integrator_weights(kw["dz"], 1, "interior").dot(graft), ww=1.0)
        with Context(BRUSH, **kw) as c:
            got.append(c.propagate_homopolymer(w))
    (want, r64), (dens, r) = got
    assert abs(np.log(r.Qsum / r64.Qsum)) < TOL
    assert np.max(np.abs(dens - want)) < TOL * np.max(np.abs(want))
