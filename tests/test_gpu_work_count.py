"""pond_last_step_work counts the scheme's stencil nodes, whichever kernel steps
the grid: one iteration from a known gauge against the windows' definition."""
import numpy as np
import pytest

from tests.states import smooth_state

pytestmark = pytest.mark.gpu

EC1, EC2 = 1.3556261799742657, 2.8569700138728056


def _work(pond, lattice, shape, interp, rho, g, precision="fp64", mask=None):
    with pond.Solver(lattice=lattice, shape=shape, interp=interp, precision=precision, tau=0.8, max_iter=1) as s:
        if mask is not None:
            s.set_mask(mask)
        s.set_state(rho, g)
        s.step(1)
        return s.last_step_work()


def _union(origins, n):
    """positions in the union of windows [o, o + n) per node; origins [classes, nodes]"""
    pos = np.sort((origins[:, None] + np.arange(n)[None, :, None]).reshape(-1, origins.shape[1]), axis=0)
    return 1 + (np.diff(pos, axis=0) != 0).sum(0)


@pytest.mark.parametrize("nx", [1000, 4096, 4097])
@pytest.mark.parametrize("interp", [2, 3, 4, 5, 7, 8])
@pytest.mark.parametrize("du", [0.3, 12.0])
def test_d1q5(pond, nx, interp, du):
    rho, g = smooth_state((nx, 1, 1), 1, seed=interp, modes=1, T0=0.3 if du < 1 else 40.0, du=du, dT=0.02)
    x = np.arange(nx)
    v = np.sqrt(g[3]) * np.array([0, EC1, -EC1, EC2, -EC2])[:, None] + g[0]
    if interp == 7:
        o = np.concatenate([np.floor(x + m * v) - 1 for m in (-2, -1, 0, 1)])
        want = (o.max(0) + 4 - o.min(0)).sum()
    elif interp == 8:
        o = np.floor(x - v + 0.5) - 2
        want = (o.max(0) + 5 - o.min(0)).sum()
    else:
        o = np.floor(x - v) - interp // 2 + 1 if interp % 2 == 0 else np.floor(x - v + 0.5) - (interp - 1) // 2
        want = _union(o, interp).sum()
    assert _work(pond, 0, (nx, 1, 1), interp, rho, g) == want


@pytest.mark.parametrize("interp", [2, 3, 4])
def test_d3q27_float64(pond, interp):
    shape = (23, 9, 7)
    rho, g = smooth_state(shape, 3, seed=interp, modes=1, T0=0.01, du=0.2, dT=0.001)  # some |u| above c
    n = np.arange(rho.size)
    pos = (n % 23, n // 23 % 9, n // 207)
    want = 1
    for ax in range(3):
        crd = pos[ax] - (np.sqrt(3 * g[3]) * np.array([0, 1, -1])[:, None] + g[ax])
        if interp % 2 == 0:
            o = np.floor(crd) - interp // 2 + 1
        else:
            o = np.floor(crd + (0.5 if ax == 0 else 0)) - (interp - 1) // 2
        want = want * _union(o, interp)
    assert _work(pond, 1, shape, interp, rho, g) == want.sum()


def test_gap2(pond):
    nx = 3000
    rho, g = smooth_state((nx, 1, 1), 1, seed=1, modes=1, T0=0.02, du=0.02, dT=0.002)
    mask = (np.arange(nx) % 3 != 0).astype(np.uint8)
    assert _work(pond, 0, (nx, 1, 1), 9, rho, g, mask=mask) == 10 * int(mask.sum())
