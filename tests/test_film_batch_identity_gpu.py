"""The first SCF iteration of a batched film and of its single context: Q and
the densities are the same bits, whatever else is in the batch, and however the
context runs its first pass."""
import numpy as np
import pytest

from adscf_gb300 import BRUSH, FILM_1D, FP64, SPLIT, MIX_SIMPLE, Batch, Context
from oracle import film as of

pytestmark = pytest.mark.gpu


def film(rng, rows, prec, brush=False, ns=70):
    gz = rows - 1
    depth = 3.0 + 0.01 * gz
    z = np.arange(rows) / gz
    dz = of.mesh_from_zr(depth * (z + 0.05 * np.sin(2 * np.pi * z) / (2 * np.pi)))
    kw = dict(grid=(1, 1, gz), size=(1.0, 1.0, depth), dz=dz, dss=of.contour_steps(ns, ds_scheme=1), n_a=ns // 3,
              block_length=(0.5, 0.5), chi=15.0, kappa=25.0, int_scheme=1, int_span=1, precision=prec,
              mixing_type=MIX_SIMPLE, lam=0.1)
    if brush:
        graft = np.exp(-0.5 * ((z - 0.1) / 0.03) ** 2)
        graft[0] = graft[-1] = 0.0
        kw.update(geometry=BRUSH, ensemble=1, rho=0.3, graft=graft, ww=1.0)
        w = (np.cos(6 * np.pi * z) + 0.1 * rng.standard_normal(rows))[None]
    else:
        kw.update(geometry=FILM_1D, ensemble=2, mu=0.4)
        w = np.stack([s * 2.0 * np.cos(6 * np.pi * z) for s in (1, -1)]) + 0.1 * rng.standard_normal((2, rows))
    w[:, 0] = w[:, -1] = 0.0
    return kw, w.reshape(-1, rows, 1, 1)


ROWS = {SPLIT: (40, 128, 129, 200, 256, 257, 700, 1501), FP64: (40, 64, 65, 128, 161, 256, 257, 384, 385, 513, 700, 1024, 1025, 2049)}


@pytest.mark.parametrize("prec,most", [(SPLIT, 4096), (FP64, 4096), (FP64, 128)])
@pytest.mark.parametrize("brush", [False, True])
def test_batch_equals_singles(rng, prec, most, brush):
    inst, w = zip(*(film(rng, r, prec, brush) for r in ROWS[prec] if r <= most))
    with Batch(list(inst)) as b:
        b.set_fields(list(w))
        rb = b.scf_run(1)
        db = b.get_densities()
    for kw, wi, r, d in zip(inst, w, rb, db):
        kw = dict(kw)
        with Context(kw.pop("geometry"), **kw) as c:
            c.set_field(wi)
            rs = c.scf_run(1)
            assert r.Qsum == rs.Qsum
            assert np.array_equal(d.ravel(), c.get_density())


@pytest.mark.parametrize("rows", [200, 501, 1001])
def test_first_pass_inside_a_capture(rng, rows):
    """The factors of FP64 lines have no memory yet when the first pass of a
    context is captured: the same bits as a pass that has."""
    torch = pytest.importorskip("torch")
    kw, w = film(rng, rows, FP64)
    kw.pop("geometry")
    got = []
    for captured in (False, True):
        with Context(FILM_1D, **kw) as c:
            s = torch.cuda.Stream()
            c._ck(c.lib.adscf_set_stream(c.h, s.cuda_stream))
            c.set_field(w)
            stages = lambda: [c._ck(c.lib.adscf_enqueue(c.h, k, 1)) for k in (1, 2, 3)]  # noqa: E731
            if captured:
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
                    stages()
                with torch.cuda.stream(s):
                    g.replay()
            else:
                stages()
            s.synchronize()
            got.append(c.get_density())
            if captured:                     # and a pass with the memory after all
                c.set_field(w)
                c.scf_run(1)
                got.append(c.get_density())
            c._ck(c.lib.adscf_set_stream(c.h, None))
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])


@pytest.mark.parametrize("rows", [41, 200, 300, 1024])
def test_lines_are_the_same_bits_in_contexts_of_more(rng, rows):
    """77 lines make their factors as they go, one line has them made ahead."""
    kw, w = film(rng, rows, FP64)
    kw.pop("geometry")
    kw.update(ensemble=1, rho=1.0)
    kw.pop("mu")
    step = []
    for lines in (1, 77):
        kw["grid"] = (lines, 1, rows - 1)
        with Context(FILM_1D, **kw) as c:
            d, r = c.propagate_diblock(np.repeat(w, lines, axis=-1))
            step.append(d.reshape(2, rows, lines) * r.Qsum)
    # density = distribution times a common factor over Q: a product rounded twice
    a, b = step[0][..., 0], step[1]
    ratio = np.max(b) / np.max(a)
    assert np.max(np.abs(b / ratio - a[..., None])) < 8 * np.finfo(float).eps * np.max(a)
