"""FP64 chains of one-line films that apply factors made ahead: row counts
around the edges of the lanes (2 to 8 rows each) and of the four warps, against
the FP64 oracle, and against the chains that eliminate as they go (contexts of
more lines than find an SM each)."""
import numpy as np
import pytest

from adscf_gb300 import BRUSH, FILM_1D, FP64, MIX_LAMBDA, Context
from oracle import film as of

pytestmark = pytest.mark.gpu

ROWS = [3, 9, 63, 64, 65, 128, 255, 256, 257, 384, 385, 512, 513, 640, 641, 768, 769, 896, 897, 1023, 1024]


def film(rows, ns):
    gz = rows - 1
    depth = 3.0 + 0.01 * gz
    zr = depth * (np.arange(rows) / gz + 0.05 * np.sin(2 * np.pi * np.arange(rows) / gz) / (2 * np.pi))
    dz = of.mesh_from_zr(zr)
    return dict(grid=(1, 1, gz), size=(1.0, 1.0, depth), dz=dz, dss=of.contour_steps(ns, ds_scheme=1), n_a=ns // 3,
                block_length=(0.5, 0.5), chi=15.0, kappa=25.0, int_scheme=1, int_span=1, ensemble=2, mu=0.4,
                precision=FP64, mixing_type=MIX_LAMBDA, lam=0.1), zr / depth


def fields(rng, z, n=2):
    w = np.stack([s * 2.0 * np.cos(6 * np.pi * z) for s in (1, -1)][:n]) + 0.1 * rng.standard_normal((n, z.size))
    w[:, 0] = w[:, -1] = 0.0
    return w


# rounding of 30 solves: 1e-16 times the matrix's O(ds / dz^2) ~ 100
@pytest.mark.parametrize("rows", ROWS)
def test_rows_vs_oracle(rng, rows):
    kw, z = film(rows, 30)
    w = fields(rng, z)
    step = lambda p, f, ds: of.cn_step_1d(p, f, kw["dz"], ds)  # noqa: E731
    ref = of.film_propagate_diblock(w, kw["dz"], kw["dss"], kw["n_a"], step, int_scheme=1, span="interior",
                                    ensemble=2, mu=0.4, sizes=kw["size"])
    with Context(FILM_1D, **kw) as c:
        dens, res = c.propagate_diblock(w.reshape(2, rows, 1, 1))
    assert abs(res.Qsum / ref["Qsum"] - 1.0) < 1e-11
    assert np.max(np.abs(dens.reshape(2, rows) - ref["density"])) < 5e-11 * np.max(np.abs(ref["density"]))


@pytest.mark.parametrize("rows,lines", [(10, 1), (200, 76), (300, 5), (1024, 2)])
@pytest.mark.parametrize("low", [0.0, -60.0, -400.0])
def test_lines_vs_more_lines(rng, rows, lines, low):
    """The same lines in a context of 77, whose chains eliminate as they go,
    with fields that leave some systems short of dominance too."""
    kw, z = film(rows, 24)
    w = np.stack([fields(rng, z) for _ in range(77)], axis=-1)          # [2][z][x]
    w[:, rows // 2, ::2] += low
    out = []
    for n in (lines, 77):
        kw["grid"] = (n, 1, rows - 1)
        with Context(FILM_1D, **kw) as c:
            for _ in range(2):      # a second pass on the kept workspace
                d, _ = c.propagate_diblock(np.ascontiguousarray(w[..., :n]).reshape(2, rows, 1, n))
            out.append(d.reshape(2, rows, n)[..., :lines] * (n if n == 77 else lines))
    a, b = out
    # densities carry the common factor exp(mu) / volume-like terms of their own context: compare shapes
    a, b = a / np.max(np.abs(a)), b / np.max(np.abs(b))
    assert np.max(np.abs(a - b)) < 5e-11


@pytest.mark.parametrize("rows", [40, 700])
def test_brush(rng, rows):
    kw, z = film(rows, 50)
    graft = np.exp(-0.5 * ((z - 0.1) / 0.03) ** 2)
    graft[0] = graft[-1] = 0.0
    w = fields(rng, z, 1)[0]
    ref = of.propagate_homopolymer(w, kw["dz"], kw["dss"], graft, 0.3, sizes=kw["size"])
    kw.update(ensemble=1, rho=0.3, graft=graft, ww=1.0)
    kw.pop("mu")
    with Context(BRUSH, **kw) as c:
        dens, res = c.propagate_homopolymer(w)
    assert abs(res.Qsum / ref["Qsum"] - 1.0) < 1e-11
    assert np.max(np.abs(dens - ref["density"])) < 1e-10 * np.max(np.abs(ref["density"]))
