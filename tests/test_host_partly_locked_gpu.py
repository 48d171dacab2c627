"""Caller arrays of which only a part is page-locked: every call that copies to
or from the host takes them, as it takes pageable arrays."""
import mmap

import numpy as np
import pytest

from adscf_gb300 import BULK, FP64, MIX_SIMPLE, Batch, Context, _lib

pytestmark = pytest.mark.gpu

N = 64                                   # 4 MiB of two species
BYTES = 2 * N ** 3 * 8


@pytest.fixture(params=["start", "end", "ends"])
def partly(request):
    """A function giving arrays of BYTES whose start, end, or both (with a gap
    between) are registered."""
    torch = pytest.importorskip("torch")
    rt = torch.cuda.cudart()
    torch.zeros(1, device="cuda")
    page = mmap.PAGESIZE
    third = BYTES // 3 // page * page
    regs, keep = [], []

    def make(values=None):
        m = mmap.mmap(-1, BYTES)
        a = np.frombuffer(m, dtype=np.float64)
        keep.append((m, a))
        for off in {"start": (0,), "end": (BYTES - third,), "ends": (0, BYTES - third)}[request.param]:
            p = a.ctypes.data + off
            assert int(rt.cudaHostRegister(p, third, 0)) == 0
            regs.append(p)
        a[:] = 0.0 if values is None else values.ravel()
        return a

    yield make
    for p in regs:
        rt.cudaHostUnregister(p)


def test_context(rng, partly):
    w = rng.standard_normal((2, N, N, N))
    kw = dict(grid=(N, N, N), size=(4.0, 4.0, 4.0), ds=0.25, precision=FP64, mixing_type=MIX_SIMPLE, lam=0.1)
    with Context(BULK, **kw) as c:
        c.set_field(w)
        c.scf_run(1)
        x, d = c.get_field(), c.get_density()
        c.set_field(partly(w))
        c.scf_run(1)
        for get, want in ((c.lib.adscf_get_field, x), (c.lib.adscf_get_density, d)):
            out = partly()
            c._ck(get(c.h, _lib.dptr(out)))
            assert np.array_equal(out, want)
        c.set_field(w)
        f, dens = partly(w), partly()
        c._ck(c.lib.adscf_scf_iteration(c.h, _lib.dptr(f), _lib.dptr(dens), None))
        assert np.array_equal(f, x) and np.array_equal(dens, d)


def test_batch(rng, partly):
    w = rng.standard_normal((2, N, N, N))
    with Batch([dict(geometry=BULK, grid=(N, N, N), size=(4.0, 4.0, 4.0), ds=0.25, precision=FP64,
                     mixing_type=MIX_SIMPLE, lam=0.1)]) as b:
        b._ck(b.lib.adscf_batch_set_fields(b.h, _lib.dptr(partly(w))))
        out = partly()
        b._ck(b.lib.adscf_batch_get_fields(b.h, _lib.dptr(out)))
        assert np.array_equal(out, w.ravel())
        f = np.zeros(1)
        b._ck(b.lib.adscf_batch_forward(b.h, _lib.dptr(partly(w)), _lib.dptr(f)))
        assert f[0] == b.forward([w])[0]
