"""Bulk batches on the mixed-radix passes, a stream per grid, against the
persistent sweep of the line passes and single contexts: grids that differ,
repeat with other contours, have one-point axes or a column tile that does not
divide x, and one-step contours."""
import numpy as np
import pytest

from adscf_gb300 import BULK, FP64, SPLIT, MIX_SIMPLE, Batch, Context

pytestmark = pytest.mark.gpu

GRIDS = [((24, 24, 24), 0.05, 0.3), ((24, 24, 24), 0.1, 0.5), ((9, 25, 27), 0.05, 0.5), ((30, 1, 40), 0.05, 0.4),
         ((1, 1, 20), 0.1, 0.5), ((64, 64, 64), 0.1, 0.5), ((16, 12, 10), 0.5, 0.5), ((24, 24, 24), 0.04, 0.25)]


def batch(prec, k=None):
    return [dict(geometry=BULK, grid=g, size=(3.3, 3.1, 2.9), ds=ds, block_length=(f, 1.0 - f), chi=15.0, kappa=20.0,
                 precision=prec, mixing_type=MIX_SIMPLE, lam=0.1) for g, ds, f in GRIDS[:k]]


# one iteration from the same field: FP64 1e-16 and FP32 6e-8 a step over at most 25 steps (the energy of
# split results with kappa = 20 on residuals of that size)
@pytest.mark.parametrize("prec,tol", [(FP64, 1e-12), (SPLIT, 2e-6)])
def test_batch_vs_sweep_and_singles(rng, prec, tol, monkeypatch):
    insts = batch(prec)
    w = [rng.standard_normal((2,) + i["grid"][::-1]) for i in insts]
    out = []
    for pin in (None, "1"):
        if pin:
            monkeypatch.setenv("ADSCF_BATCH_SWEEP", pin)
        with Batch(insts) as b:
            b.set_fields(w)
            r = b.scf_run(1)
            d1 = b.get_densities()
            b.set_fields(w)
            b.scf_run(1)
            d2 = b.get_densities()
            out.append(([v.Qsum for v in r], d1))
            assert all(np.array_equal(x, y) for x, y in zip(d1, d2))
            assert (b.lib.adscf_batch_launches(b.h) > 10) == (pin is None)
    for k, i in enumerate(insts):
        with Context(**i) as c:
            d, r = c.propagate_diblock(w[k])
        d = d.ravel()
        for q, dens in out:
            assert abs(q[k] / r.Qsum - 1.0) < tol
            assert np.max(np.abs(np.ravel(dens[k]) - d)) < 5 * tol * np.max(d)


def test_more_grids_than_streams(rng):
    """Past 64 grids the batch runs the sweep."""
    insts = [dict(batch(SPLIT, 1)[0], grid=(g, h, 8)) for g in (6, 8, 9, 10, 12, 15, 16, 18) for h in
             (5, 6, 8, 9, 10, 12, 15, 16, 18)][:65]
    with Batch(insts) as b:
        b.set_fields([np.zeros((2,) + i["grid"][::-1]) for i in insts])
        r = b.scf_run(1)
        assert b.lib.adscf_batch_launches(b.h) <= 10
    assert all(v.status == 0 for v in r)
