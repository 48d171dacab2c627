"""Gradients from kept spectra on the mixed-radix passes against the generic
reverse sweep (checkpointed, and on a pinned pass plan) and the oracle."""
import numpy as np
import pytest

from adscf_gb300 import BULK, FP64, Context

pytestmark = pytest.mark.gpu

# lines of 2, 3 and 5 factors, a column tile that does not divide x, two-dimensional and one-point axes, the
# register-FFT sizes, uneven blocks and one- and two-step contours
CASES = [((16, 12, 10), 0.05, 0.4), ((64, 64, 64), 0.05, 0.5), ((25, 27, 15), 0.1, 0.3), ((9, 1, 20), 0.05, 0.5),
         ((1, 1, 30), 0.1, 0.5), ((48, 40, 36), 0.1, 0.6), ((128, 32, 16), 0.125, 0.25), ((20, 20, 20), 0.5, 0.5),
         ((75, 8, 6), 0.1, 0.5)]


@pytest.mark.parametrize("grid,ds,f", CASES)
def test_gradient_vs_generic_sweep(rng, grid, ds, f):
    size = (3.3, 3.1, 2.9)
    w = rng.standard_normal((2,) + grid[::-1])
    kw = dict(grid=grid, size=size, ds=ds, block_length=(f, 1.0 - f), kappa=10.0, chi=15.0, precision=FP64)
    with Context(BULK, **kw) as c:
        F0 = c.forward(w)
        g0, g0b = c.backward(), c.backward()
        c.set_box((3.5, 3.0, 2.8))
        Fb = c.forward(w)
        gb = c.backward()
        c.set_adjoint_checkpoint(-1)
        Fc = c.forward(w)
        gc = c.backward()
    with Context(BULK, **kw) as c:
        c.set_pass_plan(0, 0, 0)
        F1 = c.forward(w)
        g1 = c.backward()
    assert np.array_equal(g0, g0b)
    # FP64 rounding of the chains and of sums over every frequency and step
    assert abs(F1 - F0) < 1e-12 * max(1.0, abs(F0)) and abs(Fc - Fb) < 1e-12 * max(1.0, abs(Fb))
    assert np.allclose(g1, g0, rtol=1e-10, atol=1e-12), (g0, g1)
    assert np.allclose(gc, gb, rtol=1e-10, atol=1e-12), (gb, gc)


def test_backward_after_other_calls(rng):
    """The spectra kept are those of the last forward pass."""
    grid = (24, 20, 18)
    w = rng.standard_normal((2, 2) + grid[::-1])
    kw = dict(grid=grid, size=(3.3, 3.1, 2.9), ds=0.1, block_length=(0.4, 0.6), kappa=10.0, chi=15.0, precision=FP64)
    with Context(BULK, **kw) as c:
        c.forward(w[0])
        g0 = c.backward()
        c.forward(w[1])
        c.forward(w[0])
        assert np.array_equal(c.backward(), g0)
        c.set_field(w[1])
        c.scf_run(2)
        c.forward(w[0])
        assert np.array_equal(c.backward(), g0)
        c.set_pass_plan(0, 0, 0)        # the spectra are still those of the forward pass
        assert np.array_equal(c.backward(), g0)
        c.forward(w[0])
        assert np.allclose(c.backward(), g0, rtol=1e-10, atol=1e-12)
