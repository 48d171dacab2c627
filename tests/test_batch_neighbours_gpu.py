"""A bulk instance's first iteration is the same bits whatever else is in the
batch of at most 64 grids: more instances of its grid, many other grids, or grids
whose lines the mixed-radix passes do not take."""
import numpy as np
import pytest

from adscf_gb300 import BULK, FP64, SPLIT, MIX_SIMPLE, Batch
from oracle import bulk as ob

pytestmark = pytest.mark.gpu

GRIDS = [(24, 24, 24), (32, 32, 32), (18, 20, 30), (16, 1, 40)]


def instance(grid, prec, ns=8):
    return dict(geometry=BULK, grid=grid, size=(3.7, 4.1, 3.9), ds=1.0 / ns, block_length=(0.5, 0.5), chi=15.0,
                kappa=25.0, precision=prec, mixing_type=MIX_SIMPLE, lam=0.1)


def first(inst, w):
    with Batch(inst) as b:
        b.set_fields(w)
        r = b.scf_run(1)
        return [x.Qsum for x in r], b.get_densities()


def others(kind):
    if kind == "same":
        return [g for g in GRIDS for _ in range(40)]
    if kind == "grids":
        return [(x, y, z) for x in (8, 9, 10, 12, 15) for y in (4, 5, 6, 8) for z in (3, 5, 9)]   # 60: 64 in all
    return [(1080, 2, 3), (2, 1125, 2)]


@pytest.mark.parametrize("prec", [FP64, SPLIT])
@pytest.mark.parametrize("kind", ["same", "grids", "long"])
def test_same_bits_in_any_company(rng, prec, kind):
    inst = [instance(g, prec) for g in GRIDS]
    w = [rng.standard_normal((2,) + g[::-1]) for g in GRIDS]
    q0, d0 = first(inst, w)
    more = others(kind)
    v = [rng.standard_normal((2,) + g[::-1]) for g in more]
    q1, d1 = first(inst + [instance(g, prec, 6) for g in more], w + v)
    for k in range(len(GRIDS)):
        assert q0[k] == q1[k]
        assert np.array_equal(d0[k], d1[k])
    # and the company is right: FP64 rounding of 6 steps; FP32 rounding of the non-constant modes
    for g, f, d in list(zip(more, v, d1[len(GRIDS):]))[-3:]:
        ref = ob.propagate_diblock(f, g, (3.7, 4.1, 3.9), 1.0 / 6, (0.5, 0.5))
        want = ob.density_by_type(ref["density"])
        assert np.max(np.abs(d - want)) < (1e-11 if prec == FP64 else 1e-5) * np.max(want)


@pytest.mark.parametrize("kind", ["same", "long"])
def test_gradients_in_any_company(rng, kind):
    inst = [instance(g, FP64) for g in GRIDS[:3]]
    w = [rng.standard_normal((2,) + g[::-1]) for g in GRIDS[:3]]
    more = others(kind)[:6]
    v = [rng.standard_normal((2,) + g[::-1]) for g in more]
    with Batch(inst) as b:
        f0, g0 = b.forward(w), b.backward()
    with Batch(inst + [instance(g, FP64, 6) for g in more]) as b:
        f1, g1 = b.forward(w + v), b.backward()
    assert np.array_equal(f0, f1[:3]) and np.array_equal(g0, g1[:3])
