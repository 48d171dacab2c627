"""A contour schedule with a step backwards: its systems are not diagonally
dominant whatever the field, and run the reference's recurrence.  h = 1/2 and a
step of -1/16 make the diagonal of a row with a field of 24 exactly zero (1 - 4/16
- 24/32), which the recurrence passes and an elimination that starts there does
not."""
import numpy as np
import pytest

from adscf_gb300 import FILM_1D, FILM_3D, FP64, SPLIT, Batch, Context, MIX_SIMPLE
from oracle import film as of

pytestmark = pytest.mark.gpu


def film(gz, grid=(1, 1)):
    dss = np.r_[0.0, np.full(20, 1.0 / 16)]
    dss[7] = -1.0 / 16
    return dict(grid=(*grid, gz), size=(6.0, 6.0, 0.5 * gz), dz=np.r_[0.0, np.full(gz, 0.5)], dss=dss, n_a=10,
                block_length=(0.5, 0.5), chi=15.0, kappa=25.0, int_scheme=1, int_span=1, ensemble=2, mu=0.4, precision=FP64)


def oracle(kw, w, step):
    gx, gy, _ = kw["grid"]
    return of.film_propagate_diblock(w, kw["dz"], kw["dss"], kw["n_a"], step, dx=6.0 / gx, dy=6.0 / gy, int_scheme=1,
                                     span="interior", ensemble=2, mu=0.4, sizes=kw["size"])


# one such step: its solves amplify rounding by the condition number, a few hundred
@pytest.mark.parametrize("gz", [40, 300, 600])
def test_lines(rng, gz):
    kw = film(gz)
    w = 0.1 * rng.standard_normal((2, gz + 1))
    w[:, 0] = w[:, -1] = 0.0
    w[:, 10] = w[:, 15] = 24.0
    ref = oracle(kw, w, lambda p, f, ds: of.cn_step_1d(p, f, kw["dz"], ds))
    with Context(FILM_1D, **kw) as c:
        dens, res = c.propagate_diblock(w.reshape(2, gz + 1, 1, 1))
    assert abs(res.Qsum / ref["Qsum"] - 1.0) < 1e-11
    assert np.max(np.abs(dens.reshape(2, -1) - ref["density"])) < 1e-11 * np.max(np.abs(ref["density"]))
    with Batch([dict(kw, geometry=FILM_1D, mixing_type=MIX_SIMPLE, lam=0.1)]) as b:
        b.set_fields([w.reshape(2, gz + 1, 1, 1)])
        b.scf_run(1)
        d = b.get_densities()[0]
    assert np.max(np.abs(d.reshape(2, -1) - ref["density"])) < 1e-11 * np.max(np.abs(ref["density"]))


def test_planes(rng):
    gz = 20
    kw = film(gz, (12, 10))
    w = 0.1 * rng.standard_normal((2, gz + 1, 10, 12))
    w[:, 0] = w[:, -1] = 0.0
    w[:, 3, 2, 5] = w[:, 9, 4, 7] = 24.0
    ref = oracle(kw, w, lambda p, f, ds: of.adi_step_3d(p, f, kw["dz"], 6.0 / 12, 6.0 / 10, ds))
    with Context(FILM_3D, **kw) as c:
        dens, res = c.propagate_diblock(w)
    assert abs(res.Qsum / ref["Qsum"] - 1.0) < 1e-11
    assert np.max(np.abs(dens - ref["density"])) < 1e-10 * np.max(np.abs(ref["density"]))


def test_planes_split_after_a_film_without(rng):
    """The tuner's choice for the shape was made by a film that may run the sweeps on
    lines of any length; this one may not.  FP32 rounding of the increments, 6e-8 a
    step, times the matrices' O(ds / h^2) ~ 1."""
    gz = 20
    w = 0.1 * rng.standard_normal((2, gz + 1, 10, 12))
    w[:, 0] = w[:, -1] = 0.0
    for back in (False, True, False):
        kw = dict(film(gz, (12, 10)), precision=SPLIT)
        if not back:
            kw["dss"] = np.abs(kw["dss"])
        ref = oracle(kw, w, lambda p, f, ds: of.adi_step_3d(p, f, kw["dz"], 6.0 / 12, 6.0 / 10, ds))  # noqa: B023
        with Context(FILM_3D, **kw) as c:
            dens, res = c.propagate_diblock(w)
        assert abs(res.Qsum / ref["Qsum"] - 1.0) < 2e-6
        assert np.max(np.abs(dens - ref["density"])) < 1e-5 * np.max(np.abs(ref["density"]))
