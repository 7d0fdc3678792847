"""The float32 kernels' convergence test compares the populations in float64
(isConv): a difference that float32 would round onto the other side of the
tolerance decides as the exact one does."""
import numpy as np
import pytest

from tests.states import perturbed_populations, smooth_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("interp", [2, 3, 4])
def test_population_differences_are_exact(orc, pond, interp):
    """One iteration whose populations move by factors: tolerances equal to single nodes' exact largest
    differences, which float32 rounds below or above."""
    shape = (24, 12, 8)
    rho, g = smooth_state(shape, 3, seed=interp, modes=1, du=0.03)
    rng = np.random.default_rng(interp)
    f = perturbed_populations(orc, 1, rho, g, seed=interp, eps=0.0) * rng.uniform(0.05, 4.0, (27, rho.size))
    rho, g, f = (a.astype(np.float32).astype(float) for a in (rho, g, f))

    def step(tol):
        # tau so long that the collision leaves the iterate as it is
        with pond.Solver(lattice=1, shape=shape, interp=interp, precision="fp32", tau=1e12, max_iter=1, tol_abs=tol,
                         tol_rel=0.0) as s:
            s.set_gauge_tolerance(1e30, 0.0)
            s.set_state(rho, g, f=f)
            s.step(1)
            return s.get_state()[0], s.diagnostics()["nonconverged"]

    new, nc = step(1e-7)
    assert nc == rho.size
    exact = np.abs(new - f).max(0)
    rounded = np.abs((new.astype(np.float32) - f.astype(np.float32))).max(0).astype(float)
    checked = 0
    for node in np.flatnonzero(rounded != exact)[:6]:
        for tol in (exact[node], (exact[node] + rounded[node]) / 2):
            assert step(tol)[1] == int((exact >= tol).sum())
            checked += int((rounded >= tol).sum()) != int((exact >= tol).sum())
    assert checked >= 4
