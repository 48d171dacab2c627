"""Propagation on grids of mixed-radix lines (lengths of 2, 3 and 5 factors,
unequal axes, one-point axes) against the FP64 oracle: the radices 2 to 16 and
their composites, one to several stages, planes that fit a block and planes
that do not, and the two plans of one shape against each other."""
import numpy as np
import pytest

from adscf_gb300 import BULK, FP64, SPLIT, MIX_SIMPLE, Context
from oracle import bulk as ob

pytestmark = pytest.mark.gpu

SHAPES = [(15, 16, 18), (20, 24, 27), (25, 30, 9), (36, 45, 6), (60, 72, 10), (81, 54, 5), (12, 10, 125),
          (96, 4, 100), (64, 1, 300), (300, 1, 2), (1, 1, 90), (1, 50, 40), (40, 75, 1), (150, 2, 3),
          (160, 160, 2), (180, 180, 2), (2, 1000, 3), (1000, 1, 4), (64, 32, 16), (16, 16, 16), (5, 3, 2), (8, 640, 1)]


# FP64: rounding of ~6 transforms a step over 12 steps; split: FP32 rounding of
# the non-constant modes, random over the steps
@pytest.mark.parametrize("prec,tq,tphi", [(FP64, 1e-12, 1e-11), (SPLIT, 1e-6, 1e-5)])
@pytest.mark.parametrize("grid", SHAPES)
def test_propagation_vs_oracle(rng, grid, prec, tq, tphi):
    gx, gy, gz = grid
    size, ds, f = (3.7, 4.1, 3.9), 1.0 / 12, (5 / 12, 7 / 12)
    w = rng.standard_normal((2, gz, gy, gx))
    ref = ob.propagate_diblock(w, grid, size, ds, f)
    want = ob.density_by_type(ref["density"])
    with Context(BULK, grid=grid, size=size, ds=ds, block_length=f, precision=prec) as c:
        dens, res = c.propagate_diblock(w)
        again, _ = c.propagate_diblock(w)
    assert abs(res.Qsum / ref["Qsum"] - 1.0) < tq
    assert np.max(np.abs(dens - want)) < tphi * np.max(want)
    assert np.array_equal(dens, again)


@pytest.mark.parametrize("prec", [FP64, SPLIT])
def test_box_change_and_scf_follow_the_oracle(rng, prec):
    """set_box rewrites the tables the passes read; an SCF iteration replays
    them from its graph."""
    grid, f, ds = (20, 18, 25), (0.5, 0.5), 0.1
    w = rng.standard_normal((2, 25, 18, 20))
    with Context(BULK, grid=grid, size=(3.0, 3.0, 3.0), ds=ds, block_length=f, precision=prec,
                 mixing_type=MIX_SIMPLE, lam=0.1) as c:
        c.set_field(w)
        c.scf_run(1)
        c.set_box((3.5, 4.0, 3.2))
        c.set_field(w)
        r = c.scf_run(1)
    ref = ob.propagate_diblock(w, grid, (3.5, 4.0, 3.2), ds, f)
    assert abs(r.Qsum / ref["Qsum"] - 1.0) < (1e-12 if prec == FP64 else 1e-6)


def test_default_plan_without_the_tuner_agrees(rng, monkeypatch):
    """The plane pass and the separate y passes do the same arithmetic."""
    grid, size, ds, f = (30, 36, 40), (3.7, 4.1, 3.9), 0.1, (0.4, 0.6)
    w = rng.standard_normal((2, 40, 36, 30))
    out = []
    for tune in ("1", "0"):
        monkeypatch.setenv("ADSCF_AUTOTUNE", tune)
        for prec in (FP64, SPLIT):
            with Context(BULK, grid=grid, size=size, ds=ds, block_length=f, precision=prec) as c:
                out.append(c.propagate_diblock(w)[0])
    assert np.array_equal(out[0], out[2]) and np.array_equal(out[1], out[3])


# FP64 1e-16 and FP32 6e-8 (random over the transforms' operations) per step, 20 steps
@pytest.mark.parametrize("grid,prec,tol", [((64, 64, 64), FP64, 1e-12), ((128, 64, 32), FP64, 1e-12),
                                           ((256, 32, 64), FP64, 1e-12), ((256, 32, 32), SPLIT, 2e-6),
                                           ((32, 256, 64), SPLIT, 2e-6), ((64, 32, 256), SPLIT, 2e-6),
                                           ((30, 36, 40), SPLIT, 2e-6)])
def test_against_the_line_passes(rng, grid, prec, tol):
    """Grids with a register FFT on every axis that run the mixed-radix
    passes; a pinned plan runs the line passes."""
    w = rng.standard_normal((2,) + grid[::-1])
    with Context(BULK, grid=grid, size=(3.7, 4.1, 3.9), ds=0.05, block_length=(0.4, 0.6), precision=prec) as c:
        a, ra = c.propagate_diblock(w)
        c.set_pass_plan(0, 0, 0)
        b, rb = c.propagate_diblock(w)
    assert abs(ra.Qsum / rb.Qsum - 1.0) < tol
    assert np.max(np.abs(a - b)) < 5 * tol * np.max(np.abs(b))


@pytest.mark.parametrize("grid", [(2, 1, 1), (1, 5, 1), (1, 1, 3), (3, 4, 5), (25, 1, 1), (1, 1, 125), (6, 1, 50),
                                  (30, 9, 8), (27, 20, 16), (10, 75, 12), (16, 45, 40), (32, 32, 32), (36, 30, 32)])
def test_small_fp64_grids(rng, grid):
    """One output of a butterfly per lane up to 32768 points (the last grid is
    past it): radices 2 to 5, one-point axes, butterflies that do not fill a
    warp, and columns that do not fill a tile."""
    size, ds, f = (3.7, 4.1, 3.9), 0.05, (0.4, 0.6)
    w = rng.standard_normal((2,) + grid[::-1])
    ref = ob.propagate_diblock(w, grid, size, ds, f)
    want = ob.density_by_type(ref["density"])
    with Context(BULK, grid=grid, size=size, ds=ds, block_length=f, precision=FP64) as c:
        dens, res = c.propagate_diblock(w)
        c.set_field(w)
        r = c.scf_run(1)
    # FP64 rounding of 20 steps
    assert abs(res.Qsum / ref["Qsum"] - 1.0) < 1e-12 and abs(r.Qsum / res.Qsum - 1.0) < 1e-12
    assert np.max(np.abs(dens - want)) < 5e-12 * np.max(want)
