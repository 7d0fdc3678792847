"""Nodes with a NaN gauge: the step ends, and nodes whose windows do not reach them are not touched by it.
(A NaN departure point once gave window offsets that wrapped around int, and at positions equal to the order a
walk over them that did not end.)"""
import numpy as np
import pytest

from tests.states import perturbed_populations, smooth_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,energy", [("fp32", False), ("fp64", False), ("fp32", True)])
@pytest.mark.parametrize("interp", [2, 3, 4])
def test_nan_velocity(orc, pond, interp, precision, energy):
    shape = (24, 16, 12)
    rho, g = smooth_state(shape, 3, seed=interp, modes=1, T0=0.05, du=0.02, dT=0.002)
    f = perturbed_populations(orc, 1, rho, g, seed=interp, eps=0.01)
    n = np.arange(rho.size)
    x, y, z = n % 24, n // 24 % 16, n // 384
    bad = (x == interp) & (y == interp) & (z == interp)
    more = dict(ddf_dof=2) if energy else {}
    outs = []
    for spoil in (False, True):
        with pond.Solver(lattice=1, shape=shape, interp=interp, precision=precision, tau=0.8, max_iter=20, **more) as s:
            gg = g.copy()
            if spoil:
                gg[:3, bad] = np.nan
            s.set_state(rho, gg, f=f)
            s.step(1)
            outs.append(s.get_state())
    assert not np.isfinite(outs[1][2][0, bad]).any()
    # beyond the windows, and in tiles whose gauge the node does not give
    far = (np.abs(x - interp) > 8) & (np.abs(x - interp) < 16)
    for a, b in zip(*outs):
        assert np.array_equal(a[..., far], b[..., far])
