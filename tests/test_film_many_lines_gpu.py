"""Film_1D contexts of many lines: as many as leave a thread per line ahead of
the cooperative solves, and lines that are not diagonally dominant among lines
that are, line by line against the FP64 oracle."""
import numpy as np
import pytest

from adscf_gb300 import FILM_1D, FP64, SPLIT, MIX_SIMPLE, Batch, Context, _lib
from oracle import film as of

pytestmark = pytest.mark.gpu


def film(rows, ns, prec, lines):
    gz = rows - 1
    depth = 3.0 + 0.01 * gz
    z = np.arange(rows) / gz
    dz = of.mesh_from_zr(depth * (z + 0.05 * np.sin(2 * np.pi * z) / (2 * np.pi)))
    return dict(grid=(lines, 1, gz), size=(1.0, 1.0, depth), dz=dz, dss=of.contour_steps(ns, ds_scheme=1), n_a=ns // 3,
                block_length=(0.5, 0.5), chi=15.0, kappa=25.0, int_scheme=1, int_span=1, ensemble=2, mu=0.4, precision=prec)


def fields(rng, rows, kinds):
    z = np.arange(rows) / (rows - 1)
    w = np.stack([s * 2.0 * np.cos(6 * np.pi * z) for s in (1, -1)])[..., None] + 0.1 * rng.standard_normal((2, rows, kinds))
    w[:, 0] = w[:, -1] = 0.0
    return w


def oracle(kw, w):
    step = lambda p, f, ds: of.cn_step_1d(p, f, kw["dz"], ds)  # noqa: E731
    return of.film_propagate_diblock(w, kw["dz"], kw["dss"], kw["n_a"], step, int_scheme=1, span="interior", ensemble=2,
                                     mu=0.4, sizes=(1.0, 1.0, 1.0))["density"]


# FP64: rounding of the solves, 1e-16 times the matrix's O(ds / dz^2) ~ 100;
# split: FP32 rounding of the increments; both relative to the line's own values
TOL = {FP64: 5e-11, SPLIT: 1e-5}


@pytest.mark.parametrize("prec,rows,lines,cooperative", [
    (FP64, 101, 12288, True), (FP64, 101, 12289, False), (FP64, 256, 12289, True), (FP64, 301, 6144, True),
    (FP64, 301, 6145, False), (FP64, 501, 12289, False), (FP64, 1100, 4096, True), (FP64, 1100, 4097, False),
    (SPLIT, 301, 6145, True)])
def test_number_of_lines(rng, prec, rows, lines, cooperative):
    kinds = 3
    kw = film(rows, 6, prec, lines)
    w = fields(rng, rows, kinds)
    pick = rng.integers(0, kinds, lines)
    with Context(FILM_1D, **kw) as c:
        dens, _ = c.propagate_diblock(np.ascontiguousarray(w[..., pick]).reshape(2, rows, 1, lines))
        # the cooperative solves, then the recurrence of the lines they leave; or a thread per line
        assert c.lib.adscf_stage_launches(c.h, _lib.STAGE_PROPAGATE) == (2 if cooperative else 1)
    d = dens.reshape(2, rows, lines)
    for k in range(kinds):
        want = oracle(kw, w[..., k])
        got = d[..., pick == k]
        assert np.max(np.abs(got - want[..., None])) < TOL[prec] * np.max(np.abs(want))


@pytest.mark.parametrize("prec,rows", [(FP64, 40), (FP64, 200), (FP64, 300), (FP64, 1024), (FP64, 1100), (SPLIT, 300),
                                       (SPLIT, 1100)])
@pytest.mark.parametrize("lines", [1, 5, 90])
def test_dominant_lines_beside_others(rng, prec, rows, lines):
    """Every third line has a field that leaves its systems short of dominance
    and runs the recurrence; each line is compared on its own scale."""
    ns = 12
    kw = film(rows, ns, prec, lines)
    w = fields(rng, rows, 3)
    w[:, 4::9, 0] = -1.2 / np.max(kw["dss"]) * 2.0
    with Context(FILM_1D, **kw) as c:
        for _ in range(2):
            dens, _ = c.propagate_diblock(np.ascontiguousarray(w[..., np.arange(lines) % 3]).reshape(2, rows, 1, lines))
    d = dens.reshape(2, rows, lines)
    for k in range(min(3, lines)):
        want = oracle(kw, w[..., k])
        # the recurrence of a system that is not dominant loses digits
        tol = TOL[prec] * (100.0 if k == 0 else 1.0)
        assert np.max(np.abs(d[..., k::3] - want[..., None])) < tol * np.max(np.abs(want)), k


@pytest.mark.parametrize("prec", [FP64, SPLIT])
def test_batch_with_films_that_are_not_dominant(rng, prec):
    inst, w = [], []
    for i, rows in enumerate((40, 300, 200, 301, 700, 1100)):
        kw = film(rows, 12, prec, 1)
        f = fields(rng, rows, 1)[..., 0]
        if i % 2 == 0 and (prec == FP64 or rows > 256):
            f[:, 4::9] = -1.2 / np.max(kw["dss"]) * 2.0
        inst.append(dict(kw, geometry=FILM_1D, mixing_type=MIX_SIMPLE, lam=0.1))
        w.append(f)
    with Batch(inst) as b:
        b.set_fields([f.reshape(2, -1, 1, 1) for f in w])
        r = (_lib.IterResult * len(w))()
        for _ in range(2):                    # the second run starts over
            b.set_fields([f.reshape(2, -1, 1, 1) for f in w])
            b.lib.adscf_batch_scf_run(b.h, 1, -1.0, r)
        got = b.get_densities()
    for i, (kw, f, d) in enumerate(zip(inst, w, got)):
        want = oracle(kw, f)
        tol = TOL[prec] * (100.0 if i % 2 == 0 else 1.0)
        assert np.max(np.abs(d.reshape(2, -1) - want)) < tol * np.max(np.abs(want)), i


def test_split_lines_past_the_cooperative_solves(rng):
    """4097 rows run a thread per line from an FP32 copy of the field: a line is the
    same bits in contexts of one and of three (ensemble 2: no common factor)."""
    rows, kinds = 4097, 3
    w = fields(rng, rows, kinds)
    with Context(FILM_1D, **film(rows, 6, SPLIT, kinds)) as c:
        d = c.propagate_diblock(w.reshape(2, rows, 1, kinds))[0].reshape(2, rows, kinds)
    for k in range(kinds):
        with Context(FILM_1D, **film(rows, 6, SPLIT, 1)) as c:
            one = c.propagate_diblock(np.ascontiguousarray(w[..., k]).reshape(2, rows, 1, 1))[0]
        assert np.array_equal(d[..., k], one.reshape(2, rows))
