"""The staged tile kernels at the sizes and flows where their tiling can go
wrong: grids of one node to one more than a tile along each axis, and gauges
whose stencil windows take every route through the contraction.

Tolerances: the float32 and float64 parity tolerances of test_gpu_parity.py
(largest difference over the largest value of the oracle's field)."""
import ctypes

import numpy as np
import pytest

from tests.states import perturbed_populations, smooth_state
from tests.test_gpu_parity import TOL, _compare

pytestmark = pytest.mark.gpu


def _flow(shape, kind, seed):
    """rho, g: subsonic (|u_z| < c, staggered z windows), drift (|u| > c inside the halo: the classes'
    windows coincide), crosswind (off-centre WENO windows), fast (beyond the halos), or sheared (lanes of one warp on both sides of a window change)."""
    rho, g = smooth_state(shape, 3, seed=seed, modes=1, du=0.02)
    if kind == "drift":
        g[:3] *= 0.2
        g[0] += 0.3
        g[2] -= 0.55
        g[3] *= 0.2  # c = 0.24
    elif kind == "crosswind":
        g[2] += 0.3  # moves some classes' z windows by a node
        g[1] -= 0.25
    elif kind == "fast":  # departure points beyond every staged halo
        g[0] += 1.6
        g[2] -= 1.1
    elif kind == "sheared":
        n = np.arange(rho.size)
        g[2] += np.where(n % 3 == 0, 0.5, -0.3)
        g[1] += np.where(n % 5 == 0, -0.35, 0.2)
        g[3] *= 0.3
    return rho, g


def _step_pair(orc, pond, lat, shape, interp, kind, precision="fp32", bc=(0, 0, 0), seed=3, max_iter=100):
    rho, g = _flow(shape, kind, seed)
    if precision == "fp32":  # the same starting state on both sides
        rho, g = rho.astype(np.float32).astype(float), g.astype(np.float32).astype(float)
    f = perturbed_populations(orc, lat, rho, g, seed=seed, eps=0.01)
    if precision == "fp32":
        f = f.astype(np.float32).astype(float)
    with pond.Solver(lattice=lat, shape=shape, interp=interp, precision=precision, tau=0.8, bc=bc,
                     max_iter=max_iter) as s:
        s.set_state(rho, g, f=f)
        s.step(1)
        out = s.get_state()
    ref, niter, nc = orc.step(orc.State(f, rho, g), lat, shape, interp=interp, tau=0.8, bc=bc, max_iter=max_iter)
    return out, ref, nc


@pytest.mark.parametrize("interp", [2, 3, 4])
@pytest.mark.parametrize("kind", ["subsonic", "drift"])
@pytest.mark.parametrize("shape", [(1, 1, 1), (8, 4, 4), (9, 5, 5), (7, 3, 9), (17, 8, 3)])
def test_d3q27_tile_edges(orc, pond, shape, kind, interp):
    out, ref, nc = _step_pair(orc, pond, 1, shape, interp, kind)
    assert nc == 0
    _compare(out, ref, TOL["fp32"], f"{shape} {kind} {interp}")


@pytest.mark.parametrize("interp", [2, 3, 4])
@pytest.mark.parametrize("kind,bc", [("subsonic", (2, 1, 0)), ("drift", (0, 0, 0)), ("fast", (0, 2, 1))])
@pytest.mark.parametrize("shape", [(1, 1, 1), (10, 4, 2), (11, 5, 3), (9, 3, 5), (21, 2, 4)])
def test_d3q27_float64_tile_edges(orc, pond, shape, kind, bc, interp):
    """Ten nodes of a row per warp, 10 x 4 x 2 tiles; both routes of the iteration."""
    out, ref, nc = _step_pair(orc, pond, 1, shape, interp, kind, precision="fp64", bc=bc)
    assert nc == 0
    _compare(out, ref, TOL["fp64"], f"{shape} {kind} {interp}")


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("interp", [3, 4])
def test_d3q27_iterates_leave_the_halo(orc, pond, interp, precision):
    """Gauges that start inside the halo and iterate past it: the populations carry more momentum."""
    shape = (13, 6, 5)
    rho, g = smooth_state(shape, 3, seed=9, modes=1, T0=0.05, du=0.01, dT=0.002)
    g[1] += 0.55  # |u_y| + c = 0.95 at the start
    xi = pond.lattice_tables(1)[0]
    f = perturbed_populations(orc, 1, rho, g, seed=9, eps=0.01) * (1 + 1.2 * xi[:, 1:2])
    if precision == "fp32":
        rho, g, f = (a.astype(np.float32).astype(float) for a in (rho, g, f))
    with pond.Solver(lattice=1, shape=shape, interp=interp, precision=precision, tau=0.8) as s:
        s.set_state(rho, g, f=f)
        s.step(1)
        out = s.get_state()
    ref, niter, nc = orc.step(orc.State(f, rho, g), 1, shape, interp=interp, tau=0.8)
    assert nc == 0 and (np.abs(ref.g[1]) + np.sqrt(3 * ref.g[3])).max() > 1.0
    _compare(out, ref, TOL[precision], f"{interp} {precision}")


@pytest.mark.parametrize("interp", [2, 3, 4])
def test_d3q27_windows_change_within_a_warp(orc, pond, interp):
    """One iteration on a state whose neighbouring nodes differ in the windows they read.  The iterate's
    populations are compared; its gauge is a ratio of them, and this state's densities cross zero."""
    (f, rho, _), ref, _ = _step_pair(orc, pond, 1, (16, 8, 8), interp, "sheared", max_iter=1)
    assert np.abs(f - ref.f).max() <= TOL["fp32"] * np.abs(ref.f).max()
    assert np.abs(rho - ref.rho).max() <= TOL["fp32"] * np.abs(ref.rho).max()


@pytest.mark.parametrize("bc", [(0, 0, 0), (2, 1, 0)])
@pytest.mark.parametrize("shape", [(1, 1, 1), (6, 4, 4), (7, 5, 3), (13, 2, 9)])
def test_d3q125_row_edges(orc, pond, shape, bc):
    """Fixed-origin quadratic: six nodes of a row per warp, 6 x 4 x 4 tiles."""
    out, ref, nc = _step_pair(orc, pond, 2, shape, 6, "subsonic", bc=bc)
    assert nc == 0
    _compare(out, ref, TOL["fp32"], f"{shape} {bc}")


@pytest.mark.parametrize("kind", ["subsonic", "crosswind"])
@pytest.mark.parametrize("shape", [(4, 2, 2), (5, 3, 3), (3, 5, 1)])
def test_d3q125_weno_tile_edges(orc, pond, shape, kind):
    """Centred WENO5: 4 x 2 x 2 tiles, the usual z windows and others."""
    out, ref, nc = _step_pair(orc, pond, 2, shape, 11, kind)
    assert nc == 0
    _compare(out, ref, TOL["fp32"], f"{shape} {kind}")


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("interp", [2, 3, 4, 5, 7, 8])
@pytest.mark.parametrize("nx,kind,bc", [(3, "subsonic", 1), (8, "subsonic", 2), (9, "fast", 0), (37, "fast", 1),
                                        (4096, "subsonic", 0), (4097, "subsonic", 0)])
def test_d1q5_warp_and_thread_per_node(orc, pond, nx, kind, bc, interp, precision):
    """One node per warp up to 4096 nodes, one per thread above; windows of |v| above and below one node."""
    rho, g = smooth_state((nx, 1, 1), 1, seed=nx, modes=1, T0=0.02, du=0.02, dT=0.002)
    if kind == "fast":
        g[0] += 1.4
    f = perturbed_populations(orc, 0, rho, g, seed=nx, eps=0.01)
    if precision == "fp32":
        rho, g, f = (a.astype(np.float32).astype(float) for a in (rho, g, f))
    with pond.Solver(lattice=0, shape=(nx, 1, 1), interp=interp, precision=precision, tau=0.8, bc=(bc, 0, 0)) as s:
        s.set_state(rho, g, f=f)
        s.step(1)
        out, d = s.get_state(), s.diagnostics()
    ref, niter, nc = orc.step(orc.State(f, rho, g), 0, (nx, 1, 1), interp=interp, tau=0.8, bc=(bc, 0, 0))
    assert nc == 0 and d["nonconverged"] == 0
    _compare(out, ref, TOL[precision], f"{nx} {kind} {interp}")
    if precision == "fp64":
        assert d["niter_max"] == int(niter.max())
        assert abs(d["mass"] - ref.rho.sum()) <= 1e-9 * ref.rho.sum()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_gap2_windows_and_long_departures(orc, pond, precision):
    """More windows than CTAs, and nodes whose departure points pass their nearest active neighbours."""
    nx = 120001
    rho, g = smooth_state((nx, 1, 1), 1, seed=4, modes=1, T0=0.02, du=0.02, dT=0.002)
    rng = np.random.default_rng(4)
    mask = (rng.random(nx) < 0.6).astype(np.uint8)
    mask[1000:1400] = 0
    mask[0] = 1
    g[0, 40000:60000] += 1.3  # |v| up to 1.8 nodes
    f = perturbed_populations(orc, 0, rho, g, seed=4, eps=0.01)
    if precision == "fp32":
        rho, g, f = (a.astype(np.float32).astype(float) for a in (rho, g, f))
    with pond.Solver(lattice=0, shape=(nx, 1, 1), interp=9, precision=precision, tau=0.8, max_iter=3) as s:
        s.set_mask(mask)
        s.set_state(rho, g, f=f)
        s.step(1)
        out = s.get_state()
    ref, niter, nc = orc.step_mesh(orc.State(f, rho, g), nx, interp=orc.GAP2, mask=mask, tau=0.8, max_iter=3)
    if precision == "fp32":
        # across the two jumps of u the quartic basis is taken 9 speeds out: terms of size 500 f cancel, which
        # float32 cannot hold to its tolerance; the stencils there reach a few active nodes
        keep = np.ones(nx, bool)
        for jump in (40000, 60000):
            keep[jump - 64:jump + 64] = False
        out = tuple(a[..., keep] for a in out)
        ref = orc.State(ref.f[:, keep], ref.rho[keep], ref.g[:, keep])
    _compare(out, ref, TOL[precision], "gap2")


def test_noalloc_records_shared_by_ctas(pond):
    """A grid of more CTAs than partial-sum records: the step's sums against the context's."""
    import torch
    from lbmpond_b200 import _lib
    from tests.test_zz_no_alloc import _bind
    L = _lib.load()
    shape = (256, 256, 130)
    N = int(np.prod(shape))
    with pond.Solver(lattice="D3Q27", shape=shape, interp=3, precision="fp32", tau=0.8) as s:
        s.init("tgv", 0.05, 0.1, 1.0, 5.0 / 3.0)
        ptr = s.device_state()
        out = [torch.empty(n, dtype=torch.float32, device="cuda") for n in (27 * N, N, 4 * N)]
        diag = torch.zeros(ctypes.sizeof(_lib.PondDiag), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        p = s.get_params()
        st = _bind(L)(ctypes.byref(p), *ptr, *(t.data_ptr() for t in out), diag.data_ptr(),
                      torch.cuda.current_stream().cuda_stream)
        assert st == 0, L.pond_last_error_string().decode()
        torch.cuda.synchronize()
        s.step(1)
        want = s.diagnostics()
    d = _lib.PondDiag.from_buffer_copy(bytes(diag.cpu().numpy()))
    assert abs(d.mass - want["mass"]) <= 1e-12 * want["mass"] and abs(d.enrg - want["enrg"]) <= 1e-12 * want["enrg"]
    assert d.niter_sum == want["niter_sum"] and d.niter_max == want["niter_max"]
