"""Host copies: page-locked and pageable caller memory give the same values,
for sizes on both sides of the staging chunks, single contexts and batches."""
import numpy as np
import pytest

from adscf_gb300 import BULK, FILM_1D, FP64, SPLIT, MIX_SIMPLE, Batch, Context, _lib
from oracle import film as of

pytestmark = pytest.mark.gpu


def pinned(a):
    torch = pytest.importorskip("torch")
    t = torch.empty(a.size, dtype=torch.float64, pin_memory=True)
    t.numpy()[:] = a.ravel()
    return t


@pytest.mark.parametrize("n", [8, 64, 96])     # 8 KB, 4 MB and 14 MB of two species
def test_context_copies(rng, n):
    w = rng.standard_normal((2, n, n, n))
    with Context(BULK, grid=(n, n, n), size=(4.0, 4.0, 4.0), ds=0.25, precision=SPLIT, mixing_type=MIX_SIMPLE,
                 lam=0.1) as c:
        c.set_field(w)
        assert np.array_equal(c.get_field(), w.ravel())
        c.scf_run(1)
        x, d = c.get_field(), c.get_density()
        t = pinned(w)
        c.set_field(t.numpy())
        c.scf_run(1)
        for get, want in ((c.lib.adscf_get_field, x), (c.lib.adscf_get_density, d)):
            out = pinned(np.zeros(w.size))
            c._ck(get(c.h, _lib.dptr(out.numpy())))
            assert np.array_equal(out.numpy(), want)


@pytest.mark.parametrize("kind", ["bulk", "film"])
def test_batch_copies(rng, kind):
    inst, w = [], []
    for k in range(5):
        if kind == "bulk":
            g = (8 + 4 * k, 10, 12)
            inst.append(dict(geometry=BULK, grid=g, size=(4.0, 4.0, 4.0), ds=0.1, block_length=(0.4, 0.6), chi=15.0,
                             kappa=25.0, precision=SPLIT, mixing_type=MIX_SIMPLE, lam=0.1))
            w.append(rng.standard_normal((2,) + g[::-1]))
        else:
            gz = 40 + 13 * k
            dz, _ = of.tanh_mesh(gz, 3.0)
            inst.append(dict(geometry=FILM_1D, grid=(1, 1, gz), size=(1.0, 1.0, 3.0), dz=dz,
                             dss=of.contour_steps(40, ds_scheme=1), n_a=20, block_length=(0.5, 0.5), chi=15.0,
                             kappa=25.0, int_scheme=1, int_span=1, ensemble=2, mu=0.4, precision=FP64,
                             mixing_type=MIX_SIMPLE, lam=0.1))
            w.append(0.1 * rng.standard_normal((2, gz + 1, 1, 1)))
    with Batch(inst) as b:
        b.set_fields(w)
        for a, f in zip(b.get_fields(), w):
            assert np.array_equal(a, f)
        b.scf_run(2)
        x, d = b._pack(b.get_fields()), b._pack(b.get_densities())
        t = pinned(b._pack(w))
        b._ck(b.lib.adscf_batch_set_fields(b.h, _lib.dptr(t.numpy())))   # a second start of the same run
        b.scf_run(2)
        for get, want in ((b.lib.adscf_batch_get_fields, x), (b.lib.adscf_batch_get_densities, d)):
            out = pinned(np.zeros(want.size))
            b._ck(get(b.h, _lib.dptr(out.numpy())))
            assert np.array_equal(out.numpy(), want)
