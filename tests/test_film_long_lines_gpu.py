"""Line solves of one-line films around the edges of the kernels' row counts
(one warp up to 256 rows, 4 to 32 warps up to 4096, one thread beyond),
against the FP64 oracle, and batches of mixed lengths against their single
contexts."""
import numpy as np
import pytest

from adscf_gb300 import BRUSH, FILM_1D, FP64, SPLIT, MIX_LAMBDA, Batch, Context
from adscf_gb300._lib import AdscfError
from oracle import film as of

pytestmark = pytest.mark.gpu


def film(gz, ns, prec):
    depth = 0.02 * gz
    zr = depth * (np.arange(gz + 1) / gz + 0.05 * np.sin(2 * np.pi * np.arange(gz + 1) / gz) / (2 * np.pi))
    dz = of.mesh_from_zr(zr)
    dss = of.contour_steps(ns, ds_scheme=1)
    return dict(grid=(1, 1, gz), size=(1.0, 1.0, depth), dz=dz, dss=dss, n_a=ns // 3, block_length=(0.5, 0.5),
                chi=15.0, kappa=25.0, int_scheme=1, int_span=1, ensemble=2, mu=0.4, precision=prec,
                mixing_type=MIX_LAMBDA, lam=0.1), zr / depth


def fields(rng, z, n=2):
    w = np.stack([s * 2.0 * np.cos(6 * np.pi * z) for s in (1, -1)][:n]) + 0.1 * rng.standard_normal((n, z.size))
    w[:, 0] = w[:, -1] = 0.0
    return w


# FP64: the solves' rounding, 1e-16 times the matrix's O(ds / dz^2) ~ 100 and
# 30 steps; split: FP32 rounding of the increments, 6e-8 per step, random over
# the steps, as the bound of the shorter lines' tests
ROWS = [257, 384, 512, 513, 1025, 2049, 4096, 4097]


@pytest.mark.parametrize("rows,prec,tol", [(r, FP64, 1e-11) for r in [64, 65, 129, 256] + ROWS]
                         + [(r, SPLIT, 2e-6) for r in ROWS])
def test_line_lengths_vs_oracle(rng, rows, prec, tol):
    kw, z = film(rows - 1, 30, prec)
    w = fields(rng, z)
    step = lambda p, f, ds: of.cn_step_1d(p, f, kw["dz"], ds)  # noqa: E731
    ref = of.film_propagate_diblock(w, kw["dz"], kw["dss"], kw["n_a"], step, int_scheme=1, span="interior",
                                    ensemble=2, mu=0.4, sizes=kw["size"])
    with Context(FILM_1D, **kw) as c:
        dens, res = c.propagate_diblock(w.reshape(2, rows, 1, 1))
    scale = np.max(np.abs(ref["density"]))
    assert abs(res.Qsum / ref["Qsum"] - 1.0) < tol
    assert np.max(np.abs(dens.reshape(2, rows) - ref["density"])) < 5 * tol * scale


@pytest.mark.parametrize("rows,lines", [(200, 6), (300, 6), (700, 90)])
def test_many_lines_of_one_film(rng, rows, lines):
    """Several lines per context: the warps of a line share a CTA, or (few
    lines) a cluster."""
    kw, z = film(rows - 1, 20, FP64)
    kw["grid"], kw["size"] = (lines, 1, rows - 1), (1.0, 1.0, kw["size"][2])
    w = np.stack([fields(rng, z) for _ in range(lines)], axis=-1)          # [2][z][x]
    step = lambda p, f, ds: of.cn_step_1d(p, f, kw["dz"], ds)  # noqa: E731
    ref = [of.film_propagate_diblock(w[..., i], kw["dz"], kw["dss"], kw["n_a"], step, int_scheme=1,
                                     span="interior", ensemble=2, mu=0.4, sizes=kw["size"])
           for i in (0, lines - 1)]
    with Context(FILM_1D, **kw) as c:
        dens, _ = c.propagate_diblock(w.reshape(2, rows, 1, lines))
    d = dens.reshape(2, rows, lines)
    for r, i in zip(ref, (0, lines - 1)):
        assert np.max(np.abs(d[..., i] - r["density"])) < 5e-11 * np.max(np.abs(r["density"]))


@pytest.mark.parametrize("prec", [FP64, SPLIT])
def test_batch_of_mixed_lengths_follows_singles(rng, prec):
    inst, w = [], []
    for rows in (200, 256, 257, 600, 1100, 4097):
        kw, z = film(rows - 1, 16, prec)
        inst.append(dict(kw, geometry=FILM_1D))
        w.append(fields(rng, z).reshape(2, rows, 1, 1))
    with Batch(inst) as b:
        b.set_fields(w)
        rb = b.scf_run(2)
        db = b.get_densities()
    for kw, wi, r, d in zip(inst, w, rb, db):
        with Context(**kw) as c:
            c.set_field(wi)
            rs = c.scf_run(2)
            # the same line arithmetic; the contour sums in another order
            assert abs(r.Qsum / rs.Qsum - 1.0) < 1e-11
            assert np.max(np.abs(d.ravel() - c.get_density())) < 1e-9


def test_brush_on_a_long_line(rng):
    rows, ns = 700, 60
    kw, z = film(rows - 1, ns, FP64)
    graft = np.exp(-0.5 * ((z - 0.05) / 0.01) ** 2)
    graft[0] = graft[-1] = 0.0
    w = fields(rng, z, 1)[0]
    ref = of.propagate_homopolymer(w, kw["dz"], kw["dss"], graft, 0.3, sizes=kw["size"])
    kw.update(ensemble=1, rho=0.3, graft=graft, ww=1.0)
    kw.pop("mu")
    with Context(BRUSH, **kw) as c:
        dens, res = c.propagate_homopolymer(w)
    assert abs(res.Qsum / ref["Qsum"] - 1.0) < 1e-11
    assert np.max(np.abs(dens - ref["density"])) < 1e-10 * np.max(np.abs(ref["density"]))


@pytest.mark.parametrize("gz", [8, 300])
@pytest.mark.parametrize("plane,w0", [(1, -16.0), (2, -15.0)])
def test_zero_pivots_are_those_of_the_serial_recurrence(gz, plane, w0):
    """h = 0.5, ds = 0.25: a = c = -1/2, diagonals 2, so a field of -16 at
    plane 1 (diagonal 0) or -15 at plane 2 (diagonal 1/8 = a c / 2) gives the
    recurrence an exact zero pivot; -16 at plane 2 gives the pivot -1/8 and is
    solved."""
    dz = np.r_[0.0, np.full(gz, 0.5)]
    kw = dict(grid=(1, 1, gz), size=(1.0, 1.0, 0.5 * gz), dz=dz, ds=0.25, block_length=(0.5, 0.5), precision=FP64)
    w = np.zeros(gz + 1)
    w[plane] = w0
    with Context(FILM_1D, **kw) as c:
        with pytest.raises(AdscfError) as e:
            c.propagate_step(np.ones(gz + 1), w, 0.25)
        assert e.value.code == 3
        w[:] = 0.0
        w[2] = -16.0
        q = c.propagate_step(np.ones(gz + 1), w, 0.25)
    assert np.max(np.abs(q - of.cn_step_1d(np.ones(gz + 1), w, dz, 0.25))) < 1e-12 * np.max(np.abs(q))
