"""The float64 D3Q27 step where the gauge jumps by orders of magnitude within a
tile: the staged tiles pass through the gauge of the tile's centre, which costs
digits that float64 results must not lose."""
import numpy as np
import pytest

from tests.states import perturbed_populations

pytestmark = pytest.mark.gpu

# One iteration at nodes whose windows hold gauges within 1 % of their own: a
# direct transfer is a sum of 27 x 64 terms of the size of its result.
TOL = 1e-12


@pytest.mark.parametrize("interp", [2, 3, 4])
@pytest.mark.parametrize("kind", ["T 100", "T 1000", "T 10000", "u"])
def test_contrast_within_a_tile(orc, pond, kind, interp):
    """Tiles of ten nodes with their centre in another gas than the nodes x % 20 = 0."""
    shape = (40, 8, 4)
    x = np.arange(int(np.prod(shape))) % 20
    core = (x >= 3) & (x <= 8)
    rng = np.random.default_rng(interp)
    T = np.full(x.size, 0.02 ** 2 / 3)
    u = np.zeros(x.size)
    if kind == "u":
        u = np.where(core, 0.4, -0.4)
    else:
        T = np.where(core, 0.08, 0.08 / float(kind.split()[1]))
    T *= 1 + 0.01 * rng.uniform(-1, 1, x.size)
    g = np.stack([u, 0 * u, 0 * u, T])
    g[:3] += 0.01 * np.sqrt(3 * T) * rng.uniform(-1, 1, (3, x.size))
    rho = 1 + 0.02 * rng.standard_normal(x.size)
    f = perturbed_populations(orc, 1, rho, g, seed=interp, eps=0.01)
    with pond.Solver(lattice=1, shape=shape, interp=interp, precision="fp64", tau=0.8, max_iter=1) as s:
        s.set_state(rho, g, f=f)
        s.step(1)
        got = s.get_state()
    ref, _, _ = orc.step(orc.State(f, rho, g), 1, shape, interp=interp, tau=0.8, max_iter=1)
    keep = (x == 0) | (x == 5) | (x == 6)
    assert np.abs(got[0] - ref.f)[:, keep].max() <= TOL * np.abs(ref.f[:, keep]).max()
    assert np.abs(got[1] - ref.rho)[keep].max() <= TOL * np.abs(ref.rho[keep]).max()
