"""F of adscf_forward on a film is rounded once: central differences over a wall
potential's every plane (F is linear in it) meet the gradient to the last
place of F."""
import numpy as np
import pytest

from adscf_gb300 import FILM_1D, Context
from oracle import film as of
from oracle import interactions as oi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ensemble", [1, 2])
def test_differences_of_f(ensemble, rng):
    gz, depth = 40, 3.0
    dz, zr = of.tanh_mesh(gz, depth)
    ext = np.stack([a * oi.wall_potential_shape(zr, depth, 0.4) for a in (0.6, -0.3)])
    z = zr / depth
    w = np.stack([1.5 * np.cos(2 * np.pi * z), -1.5 * np.cos(2 * np.pi * z)]) + 0.1 * rng.standard_normal((2, gz + 1))
    w[:, 0] = w[:, -1] = 0.0

    def F(e):
        with Context(FILM_1D, grid=(1, 1, gz), size=(1.0, 1.0, depth), ds=0.02, block_length=(0.5, 0.5), dz=dz, kappa=25.0,
                     chi=15.0, ext_potential=e, int_scheme=1, int_span=1, ensemble=ensemble, mu=0.4) as c:
            f = c.forward(w)
            return f, c.backward_surface()[1]

    f0, dU = F(ext)
    d = 1e-5
    for c in (0, 1):
        for k in range(1, gz):
            e = [ext.copy(), ext.copy()]
            e[0][c, k] += d
            e[1][c, k] -= d
            fd = F(e[0])[0] - F(e[1])[0]
            # half a unit of each F, and of the perturbed potentials
            assert abs(fd - 2 * d * dU[c, k]) <= 1.02 * np.spacing(abs(f0)) + 4e-16 * abs(dU[c, k]), (c, k)
