"""The device buffer of a batch's host copies is bounded, and batches larger than
it are copied in turns."""
import numpy as np
import pytest

from adscf_gb300 import BULK, SPLIT, MIX_SIMPLE, Batch, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pin", [False, True])
def test_batch_larger_than_the_buffer(rng, pin):
    torch = pytest.importorskip("torch")
    inst = [dict(geometry=BULK, grid=(n, n, n), size=(4.0, 4.0, 4.0), ds=0.5, precision=SPLIT, mixing_type=MIX_SIMPLE,
                 lam=0.1) for n in (160, 30, 128, 160, 48, 160, 20)]      # 257 MB of fields
    with Batch(inst) as b:
        n = b.offsets[-1]
        w, out = (torch.empty(n, dtype=torch.float64, pin_memory=pin) for _ in range(2))
        w.numpy()[:] = rng.standard_normal(n)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        b._ck(b.lib.adscf_batch_set_fields(b.h, _lib.dptr(w.numpy())))
        b._ck(b.lib.adscf_batch_get_fields(b.h, _lib.dptr(out.numpy())))
        held = free - torch.cuda.mem_get_info()[0]
        assert np.array_equal(w.numpy(), out.numpy())
        b.scf_run(1)
        b._ck(b.lib.adscf_batch_get_densities(b.h, _lib.dptr(out.numpy())))
        assert np.all(np.isfinite(out.numpy()))
    assert held <= (136 << 20), held
