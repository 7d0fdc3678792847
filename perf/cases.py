"""The work the step library is timed on, through its public entry points.

A case is a state a program holds (on the device, or in pinned host memory
for the host-buffer pipeline) and the steps it asks for.  Except for the
batched tubes, whose state lives inside the batch, every pass starts from the
same state: a pass writes it into the solver's device buffers and steps, so
passes are comparable however often they are repeated.

Grid arrays are [..., z, y, x]; populations are in the library's order.
"""
import math

import numpy as np
import torch

import lbmpond_b200 as pond
from lbmpond_b200.batch import Batch

LAGR3, LAGR4, FIXED3, TVD, WENO5, GAP2, WENO5_ROW = 3, 4, 6, 7, 8, 9, 11
BCS = {"p": "periodic", "c": "clamp", "m": "mirror", "i": "inflow"}


def _grid(name, path, shape, interp, state, tau, steps, precision="fp32", bc="ppp"):
    nx, ny, nz = shape
    return dict(name=name, path=path, nx=nx, ny=ny, nz=nz, interp=interp, state=state, tau=tau, steps=steps,
                precision=precision, bc=bc)


def listed():
    return [
        # the benchmark: spherical Riemann problem, cubic Lagrange, the largest single grid
        _grid("sphere_256", "d3q27", (256, 256, 256), LAGR4, "blast", 0.52, 1),
        # the compressible Taylor-Green vortex, quadratic Lagrange, every node iterating
        _grid("tgv_128", "d3q27", (128, 128, 128), LAGR3, "vortex", 0.51, 1),
        # a small periodic box, as in parameter scans: few CTAs, launches and latency count
        _grid("box_32", "d3q27", (32, 32, 32), LAGR4, "vortex", 0.8, 8),
        # a ragged box between walls: mirror in x, zero gradient in y, sizes off every tile
        _grid("walls_61x45x37", "d3q27", (61, 45, 37), LAGR4, "vortex", 0.6, 2, bc="mcp"),
        # the reference's double precision and tolerances
        _grid("double_48", "d3q27", (48, 48, 48), LAGR4, "blast", 0.52, 1, precision="fp64"),
        # a gamma = 1.4 gas: energy populations beside f
        _grid("gamma14_64", "energy", (64, 64, 64), LAGR3, "vortex", 0.51, 2),
        # Mach 1.5 shock and vortex on D3Q125, centred WENO5, inflow and outflow along x
        _grid("shock_weno_48", "d3q125", (48, 48, 48), WENO5_ROW, "shock", 0.9, 1, bc="ipp"),
        # the same flow with the reference's own D3Q125 scheme (fixed-origin quadratic)
        _grid("shock_quad_96", "d3q125", (96, 96, 96), FIXED3, "shock", 0.9, 1, bc="ipp"),
        # the Sod tube of 1000 nodes in double precision with the limited scheme: many tiny steps
        _grid("tube_1000", "d1q5", (1000, 1, 1), TVD, "tube", 0.55, 50, precision="fp64", bc="ccc"),
        # a long 1D grid with every other node of its smooth stretches switched off
        _grid("mesh_4m", "mesh", (4194304, 1, 1), GAP2, "tube", 0.9, 4),
        # independent tubes of uneven length advanced together, fields read at the end
        dict(name="batch_1024", path="batch", problems=1024, lmin=256, lmax=4096, interp=WENO5, tau=0.9, steps=200),
        # states that live in host memory: copies in, one step, rho and gauge back, several in a row
        _grid("host_96", "host", (96, 96, 96), LAGR4, "blast", 0.52, 1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["d3q27", "d3q27", "d3q27", "walls", "double", "energy", "weno", "quad", "d1q5", "mesh", "batch",
                       "host"])
    tau = round(rng.uniform(0.51, 0.9), 3)

    def box(lo, hi):
        e = _log(rng, lo, hi)
        return tuple(max(lo, min(hi, int(e * rng.uniform(0.75, 1.25)))) for _ in range(3))

    if kind in ("d3q27", "walls"):
        shape = box(24, 250 if kind == "d3q27" else 96)
        steps = 1 if shape[0] * shape[1] * shape[2] > 300000 else rng.choice([2, 4, 8])
        bc = "ppp" if kind == "d3q27" else "".join(rng.choice("pcm") for _ in range(3))
        state = rng.choice(["blast", "vortex"]) if kind == "d3q27" else "vortex"
        c = _grid("", "d3q27", shape, rng.choice([2, 3, 4, 4]), state, tau, steps, bc=bc)
    elif kind == "double":
        c = _grid("", "d3q27", box(16, 56), rng.choice([3, 4]), rng.choice(["blast", "vortex"]), tau, 1,
                  precision="fp64")
    elif kind == "energy":
        c = _grid("", "energy", box(24, 80), rng.choice([3, 4]), "vortex", tau, 2)
    elif kind == "weno":
        c = _grid("", "d3q125", box(16, 52), WENO5_ROW, "shock", 0.9, 1, bc="ipp")
    elif kind == "quad":
        c = _grid("", "d3q125", box(16, 110), FIXED3, "shock", 0.9, 1, bc="ipp")
    elif kind == "d1q5":
        c = _grid("", "d1q5", (_log(rng, 200, 4000), 1, 1), TVD, "tube", tau, rng.choice([20, 50, 100]),
                  precision=rng.choice(["fp64", "fp32"]), bc="ccc")
    elif kind == "mesh":
        c = _grid("", "mesh", (_log(rng, 20000, 4000000), 1, 1), GAP2, "tube", tau, 4)
    elif kind == "batch":
        c = dict(path="batch", problems=_log(rng, 64, 1024), lmin=256, lmax=rng.choice([1024, 4096]), interp=WENO5,
                 tau=tau, steps=rng.choice([50, 100, 200]))
    else:
        c = _grid("", "host", box(32, 100), LAGR4, "blast", tau, 1)
    c.pop("name", None)
    return c


# ---------------------------------------------------------------- lattices

EC1, EC2 = 1.3556261799742657, 2.8569700138728056
XI = {3: (0.0, 1.0, -1.0), 5: (0.0, EC1, -EC1, EC2, -EC2)}
W1 = {3: (2 / 3, 1 / 6, 1 / 6)}
W1[5] = ((3 - (EC1 ** 2 + EC2 ** 2) + EC1 ** 2 * EC2 ** 2) / (EC1 ** 2 * EC2 ** 2),
         (EC2 ** 2 - 3) / (2 * EC1 ** 2 * (EC2 ** 2 - EC1 ** 2)),
         (EC2 ** 2 - 3) / (2 * EC1 ** 2 * (EC2 ** 2 - EC1 ** 2)),
         (EC1 ** 2 - 3) / (2 * EC2 ** 2 * (EC1 ** 2 - EC2 ** 2)),
         (EC1 ** 2 - 3) / (2 * EC2 ** 2 * (EC1 ** 2 - EC2 ** 2)))
# population of class (cx, cy, cz), classes {0, +, -} per axis, index 9 cx + 3 cy + cz
ORDER27 = (0, 3, 16, 2, 6, 18, 12, 13, 24, 1, 5, 17, 4, 7, 19, 14, 15, 25, 8, 10, 22, 9, 11, 23, 20, 21, 26)
INFLOW_T = 0.05


def _lattice(case):
    """(speeds per axis, dimensions, TLat, population of each tensor class)"""
    if case["path"] in ("d1q5", "mesh", "batch"):
        return 5, 1, 1.0, tuple(range(5))
    if case["path"] == "d3q125":
        return 5, 3, 1.0, tuple(range(125))
    return 3, 3, 1.0 / 3.0, ORDER27


def _weights(q1, dim):
    w = W1[q1]
    if dim == 1:
        return list(w)
    return [a * b * c for a in w for b in w for c in w]


def _inflow():
    """rho, ux, uy, uz, T upstream of the Mach 1.5 shock"""
    return (1.0, 1.5 * math.sqrt(5.0 / 3.0 * INFLOW_T), 0.0, 0.0, INFLOW_T)


# ---------------------------------------------------------------- states

def _fields(case, seed):
    """rho [z, y, x] and the gauge [4, z, y, x] in float64 on the GPU, from the seed."""
    rng = np.random.RandomState(seed % (1 << 31))
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dev, dt = torch.device("cuda"), torch.float64
    x = ((torch.arange(nx, device=dev, dtype=dt) + 0.5) / nx)[None, None, :]
    y = ((torch.arange(ny, device=dev, dtype=dt) + 0.5) / ny)[None, :, None]
    z = ((torch.arange(nz, device=dev, dtype=dt) + 0.5) / nz)[:, None, None]
    two_pi = 2 * math.pi

    def wave(amp, modes=2):
        t = 0.0
        for _ in range(modes):
            k = rng.randint(-2, 3, 3)
            t = t + amp * torch.sin(two_pi * (float(k[0]) * x + float(k[1]) * y + float(k[2]) * z)
                                    + rng.uniform(0, two_pi))
        return t

    if case["state"] == "blast":
        # a blast some time after the release: uniform gas outside the front, an expanding shell inside
        cx, cy, cz = rng.uniform(0.48, 0.52, 3)
        dx, dy, dz = x - cx, y - cy, z - cz
        r = torch.sqrt(dx * dx + dy * dy + dz * dz)
        edge = 0.47 * (1 + 0.02 * torch.sin(3 * torch.atan2(dy, dx + 1e-9 * (dz + 1))) + rng.uniform(-0.02, 0.02))
        s = (r / edge).clamp(max=1.0)
        env = (1 - s * s) ** 2 * (s < 1)
        shell = torch.exp(-((s - 0.75) / 0.12) ** 2) * (1 - s ** 8) * (s < 1)
        rho = 0.125 + 0.25 * env + 0.15 * shell
        T = 0.05 + 0.012 * env * (1 + 0.2 * wave(1.0)) + 0.008 * shell
        ur = (0.25 * shell + 0.1 * s * env) * (1 + 0.1 * wave(1.0)) / (r + 1e-12)
        return rho, torch.stack([ur * dx, ur * dy, ur * dz, T])
    if case["state"] == "vortex":
        t0 = 1.0 / 12.0
        u0 = 0.5 * math.sqrt(5.0 / 3.0 * t0)
        px, py, pz = (two_pi * (a + p) for a, p in zip((x, y, z), rng.uniform(0, 1, 3)))
        ux = u0 * torch.sin(px) * torch.cos(py) * torch.cos(pz) + wave(0.004)
        uy = -u0 * torch.cos(px) * torch.sin(py) * torch.cos(pz) + wave(0.004)
        uz = wave(0.01) + 0 * ux
        pr = u0 * u0 / 16 * (torch.cos(2 * px) + torch.cos(2 * py)) * (torch.cos(2 * pz) + 2) / t0
        T = t0 * (1 + 0.4 * pr) * (1 + wave(0.005))
        return (1 + pr) * (1 + wave(0.005)), torch.stack([ux, uy, uz, T])
    if case["state"] == "shock":
        # Mach 1.5 normal shock at x = 0.5 over two nodes, an isentropic vortex upstream
        ga, mach, t1 = 5.0 / 3.0, 1.5, INFLOW_T
        c1 = math.sqrt(ga * t1)
        u1 = mach * c1
        r21 = (ga + 1) * mach ** 2 / ((ga - 1) * mach ** 2 + 2)
        p21 = 1 + 2 * ga / (ga + 1) * (mach ** 2 - 1)
        eps, rad = rng.uniform(0.25, 0.35), rng.uniform(0.05, 0.08)
        dx, dy = x - rng.uniform(0.22, 0.28), y - rng.uniform(0.45, 0.55)
        e = torch.exp(0.5 * (1 - (dx * dx + dy * dy) / rad ** 2)) + 0 * z
        post = 0.5 * (1 + torch.tanh((x - 0.5) * nx / 2.0)) * (x > 0.5 - 16.0 / nx)
        pre = 1 - post
        th = 1 - (ga - 1) / 2 * (eps * e * pre) ** 2
        ux = pre * u1 + post * (u1 / r21) - eps * c1 * dy / rad * e * pre
        uy = eps * c1 * dx / rad * e * pre
        T = (pre * t1 + post * t1 * p21 / r21) * th
        rho = (pre + post * r21) * th ** (1 / (ga - 1))
        return rho + 0 * e, torch.stack([ux + 0 * e, uy, 0 * e, T])
    # tube: shocks and contacts over a few nodes, smooth waves between them
    rho, T, u = torch.ones_like(x), torch.full_like(x, 0.009), torch.zeros_like(x)
    for x0 in rng.uniform(0.1, 0.9, 3):
        s = torch.tanh((x - x0) * nx / 3.0)
        rho = rho * (1 + 0.25 * rng.uniform(0.5, 1) * s)
        T = T * (1 + 0.05 * rng.uniform(0.5, 1) * s)
    for k in (1, 2, 5):
        u = u + 0.004 * torch.sin(two_pi * k * max(1, nx // 100000) * x + rng.uniform(0, two_pi))
    return rho, torch.stack([u, 0 * u, 0 * u, T])


def _state(case, seed):
    """f [Q, N], rho [N], g [4, N] on the GPU in the case's precision: near equilibrium, as after a collision."""
    q1, dim, _, order = _lattice(case)
    rho, g = _fields(case, seed)
    rng = np.random.RandomState((seed * 7 + 3) % (1 << 31))
    t = torch.float64 if case["precision"] == "fp64" else torch.float32
    n = rho.numel()
    dev_T = g[3] - g[3].flatten()[0]  # non-equilibrium only where the field varies
    bump = dev_T / (dev_T.abs().max() + 1e-300)
    f = torch.empty((len(order), n), dtype=t, device=rho.device)
    w = _weights(q1, dim)
    for cls, q in enumerate(order):
        f[q] = (w[cls] * rho * (1 + 0.01 * rng.uniform(-1, 1) * bump)).reshape(-1).to(t)
    return f, rho.reshape(-1).to(t), g.reshape(4, -1).to(t).contiguous()


def _mask(case, seed):
    """Active nodes of the mesh: all near the steep places, every other one elsewhere."""
    rho, _ = _fields(case, seed)
    rho = rho.reshape(-1)
    steep = (rho - rho.roll(1)).abs() > 1e-3 * rho
    near = torch.nn.functional.max_pool1d(steep.float()[None, None], 33, 1, 16)[0, 0] > 0
    return near | (torch.arange(rho.numel(), device=rho.device) % 2 == 0)


class _Pointer:
    """A device array of a solver's, for torch; a tensor on it keeps the solver."""

    def __init__(self, solver, ptr, shape, precision):
        self.solver = solver
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "version": 3,
                                         "typestr": "<f8" if precision == "fp64" else "<f4"}


class _Device:
    """A solver and torch views of its two sets of device buffers."""

    def __init__(self, case, **more):
        lattice = {"d1q5": "D1Q5", "mesh": "D1Q5", "d3q125": "D3Q125"}.get(case["path"], "D3Q27")
        self.case = case
        self.solver = pond.Solver(lattice=lattice, shape=(case["nx"], case["ny"], case["nz"]), interp=case["interp"],
                                  precision=case["precision"], tau=case["tau"], bc=tuple(BCS[b] for b in case["bc"]),
                                  **more)
        self.solver.init("uniform", 1.0, 0.0, 0.0, 0.0, 0.1)
        if "i" in case["bc"]:
            self.solver.set_inflow(*_inflow())
        self.stream = torch.cuda.ExternalStream(self.solver.stream())
        self.views = {}

    def arrays(self):
        f, r, g = self.solver.device_state()
        if f not in self.views:
            s = self.solver
            self.views[f] = tuple(torch.as_tensor(_Pointer(s, p, shape, self.case["precision"]), device="cuda")
                                  for p, shape in ((f, (s.Q, s.N)), (r, (s.N,)), (g, (4, s.N))))
        return self.views[f]


def _host_case(case):
    return dict(case, path="d3q27")


def _tubes(case, seed):
    """lengths and the concatenated rho, u, T of independent Riemann tubes whose jumps span a few nodes"""
    p = case["problems"]
    lengths = np.random.default_rng(p).integers(case["lmin"], case["lmax"] + 1, p).astype(np.int32)
    rng = np.random.default_rng(seed)
    rho = np.exp(rng.uniform(-0.5 * math.log(4.0), 0.5 * math.log(4.0), (p, 2)))
    T = 0.09 * np.exp(rng.uniform(-0.5 * math.log(1.5), 0.5 * math.log(1.5), (p, 2)))
    u = 0.06 * rng.uniform(-1, 1, (p, 2))
    prob = np.repeat(np.arange(p), lengths)
    first = np.repeat(np.cumsum(lengths) - lengths, lengths)
    x = np.arange(prob.size) - first
    s = 0.5 * (1 + np.tanh((x - lengths[prob] / 2) / 4.0))
    return lengths, *(a[prob, 0] * (1 - s) + a[prob, 1] * s for a in (rho, u, T))


def prepare(case, seed):
    path = case["path"]
    if path == "batch":
        lengths, rho, u, T = _tubes(case, seed)
        b = Batch(lengths, interp=case["interp"], tau=case["tau"])
        b.set_state(rho, u, T)
        return {"batch": b, "steps": case["steps"]}
    if path == "host":
        members = []
        for k in range(3):
            host = [t.cpu().pin_memory() for t in _state(_host_case(case), seed * 3 + k)]
            members.append((host, torch.empty_like(host[1]).pin_memory(), torch.empty_like(host[2]).pin_memory()))
        d = _Device(_host_case(case))
        return {"host": d.solver, "members": members}
    if path == "energy":
        f, rho, g = _state(case, seed)
        base, d = _Device(case, ddf_dof=2), _Device(case, ddf_dof=2)
        base.solver.set_state(*(t.double().cpu().numpy() for t in (rho, g, f)))  # h at equilibrium
        return {"device": d, "base": base.solver, "steps": case["steps"]}
    d = _Device(case)
    if path == "mesh":
        d.solver.set_mask(_mask(case, seed).cpu().numpy())
    d.arrays()
    state = _state(case, seed)
    torch.cuda.synchronize()  # the solver's stream reads it
    return {"device": d, "state": state, "steps": case["steps"]}


def run(state):
    if "batch" in state:
        state["batch"].run(state["steps"])
        return state["batch"].get_state()
    if "host" in state:
        s = state["host"]
        for (f, rho, g), rho_out, g_out in state["members"]:
            s.step_host(f.data_ptr(), rho.data_ptr(), g.data_ptr(), rho_out.data_ptr(), g_out.data_ptr())
        s.sync()
        return [(rho_out, g_out) for _, rho_out, g_out in state["members"]]
    d = state["device"]
    if "base" in state:
        d.solver.copy_state_from(state["base"])
    else:
        with torch.cuda.stream(d.stream):
            for to, t in zip(d.arrays(), state["state"]):
                to.copy_(t)
    d.solver.step(state["steps"])
    d.solver.diagnostics()  # the totals a program looks at after a run of steps
    return d.arrays()


def work(case):
    """One read and one write of the state a step; two evaluations of every node's
    populations (a node that changes at all needs them), each the transfer of the
    stencil into the node's gauge contracted axis by axis."""
    if case["path"] == "batch":
        n = case["problems"] * (case["lmin"] + case["lmax"]) / 2
        return {"bytes": 2.0 * n * 8 * 4, "flops": 2.0 * case["steps"] * n * 5 * 5 * 5 * 2}
    q1, dim, _, order = _lattice(case)
    n = case["nx"] * case["ny"] * case["nz"]
    q = len(order)
    elem = 8 if case["precision"] == "fp64" else 4
    k = {TVD: 4, FIXED3: 3, GAP2: 2, WENO5_ROW: 5}.get(case["interp"], case["interp"])
    if dim == 1:
        flops = 2 * k * q * q1
    else:
        flops = 2 * q * q1 * (k ** 3 + k ** 2 + k)
    members = 3 if case["path"] == "host" else 1
    per = (2 * q if case["path"] == "energy" else q) + 5
    flops *= 2 if case["path"] == "energy" else 1
    return {"bytes": 2.0 * per * elem * n * case["steps"] * members, "flops": 2.0 * flops * n * case["steps"] * members}


# ---------------------------------------------------------------- the step in 64 bits

def _basis(q1, i, y):
    """Lagrange basis i of the speed set, at y"""
    xi = XI[q1]
    t = 1.0
    for k in range(q1):
        if k != i:
            t = t * ((y - xi[k]) / (xi[i] - xi[k]))
    return t


def _lagrange(n, s):
    """weights of n nodes 0..n-1 at s"""
    out = []
    for j in range(n):
        t = torch.ones_like(s)
        for p in range(n):
            if p != j:
                t = t * ((s - p) / (j - p))
        out.append(t)
    return out


def _padded(a, ax, bc, h, ghost=None):
    """one axis (0 = x) with h nodes on both sides; returns the array and the mirrored positions"""
    dim = a.dim() - 1 - ax
    n = a.shape[dim]
    p = torch.arange(-h, n + h, device=a.device)
    if bc == "m":
        rev = (p < 0) | (p >= n)
        idx = torch.where(p < 0, -1 - p, torch.where(p >= n, 2 * n - 1 - p, p)) % n
    else:
        rev = torch.zeros_like(p, dtype=torch.bool)
        idx = p % n if bc == "p" else p.clamp(0, n - 1)
    out = a.index_select(dim, idx)
    if ghost is not None:
        out.narrow(dim, 0, h).copy_(ghost.expand_as(out.narrow(dim, 0, h)))
    sign = torch.where(rev, -1.0, 1.0).to(a.dtype)
    return out, sign.reshape([-1] + [1] * ax)


def _weno_blend(S, u, d):
    d0, d2 = (d * d - 3 * d + 2) / 12, (d * d + 3 * d + 2) / 12
    b = [13 / 12 * (u[j] - 2 * u[j + 1] + u[j + 2]) ** 2 + 0.25 * (a * u[j] + m * u[j + 1] + c * u[j + 2]) ** 2
         for j, (a, m, c) in enumerate(((1, -4, 3), (1, 0, -1), (3, -4, 1)))]
    w = [x / (1e-6 + y) ** 2 for x, y in zip((d0, 1 - d0 - d2, d2), b)]
    return (w[0] * S[0] + w[1] * S[1] + w[2] * S[2]) / (w[0] + w[1] + w[2])


def _converge(evaluate, U, T, most=80):
    """The fixed point of the gauge: evaluate(U, T) -> populations, new U, new T."""
    old = None
    for _ in range(most):
        acc, Un, Tn = evaluate(U, T)
        Tn = torch.where(Tn < 0, T, Tn)
        step = max(float((Un - U).abs().max()), float((Tn - T).abs().max()),
                   1.0 if old is None else float((acc[0] - old).abs().max()))
        U, T, old = Un, Tn, acc[0]
        if step < 1e-13:
            break
    return acc, U, T


def _exact3d(case, f, rho, g, h=None, dof=0):
    """One step on a 3D lattice, [q, z, y, x] float64; returns f, rho, g (and h)."""
    q1, _, tlat, order = _lattice(case)
    xi, w = XI[q1], _weights(q1, 3)
    n, interp = (case["nz"], case["ny"], case["nx"]), case["interp"]
    weno = interp == WENO5_ROW
    k = 3 if interp == FIXED3 or weno else interp
    bc = case["bc"]
    halo = 6
    U, T = g[:3].clone(), g[3].clone()
    take = torch.tensor(order, device=f.device)
    sets = [(d[take], [wi * (_inflow()[0]) for wi in w]) for d in ([f] if h is None else [f, h])]
    # padded sources: populations by class, velocity, and c with the sign each axis sees
    u, c = g[:3], torch.sqrt(g[3].abs() / tlat) * torch.sign(g[3])
    us, cs = [u[a] for a in range(3)], [c, c, c]
    srcs = [s[0] for s in sets]
    for ax in range(3):
        inflow = bc[ax] == "i"
        gh = (lambda v: torch.tensor(v, dtype=f.dtype, device=f.device)) if inflow else None
        for a in range(3):
            us[a], sg = _padded(us[a], ax, bc[ax], halo, gh(_inflow()[1 + a]) if inflow else None)
            cs[a], _ = _padded(cs[a], ax, bc[ax], halo, gh(math.sqrt(_inflow()[4] / tlat)) if inflow else None)
            if a == ax:
                us[a], cs[a] = us[a] * sg, cs[a] * sg
        srcs = [_padded(s, ax, bc[ax], halo, gh(sets[i][1]).reshape(-1, 1, 1, 1) if inflow else None)[0]
                for i, s in enumerate(srcs)]

    def cut(a, o):  # the source at offset (ox, oy, oz)
        return a[..., halo + o[2]:halo + o[2] + n[0], halo + o[1]:halo + o[1] + n[1], halo + o[0]:halo + o[0] + n[2]]

    def contract(M, s, axis):
        out = torch.empty_like(s)
        for i in range(q1):
            t = out.select(axis, i)
            torch.mul(s.select(axis, 0), M[i][0], out=t)
            for b in range(1, q1):
                t.addcmul_(s.select(axis, b), M[i][b])
        return out

    def evaluate(U, T):
        C = torch.sqrt(T / tlat)
        org, wt, dist = [], [], None
        for ax in range(3):
            o, ws = [], []
            for i in range(q1):
                s = -(C * xi[i] + U[ax])
                if weno:
                    m = torch.floor(s + 0.5)
                    o.append(m - (2 if ax == 0 else 1))
                    ws.append([_lagrange(3, s - (m - 2 + j)) for j in range(3)] if ax == 0
                              else _lagrange(3, s - (m - 1)))
                    if ax == 0:
                        dist = (dist or []) + [s - m]
                    continue
                if interp == FIXED3:
                    b = torch.full_like(s, -1.0)
                elif interp % 2 == 0:
                    b = torch.floor(s) - interp // 2 + 1
                else:
                    b = (torch.floor(s + 0.5) if ax == 0 else torch.floor(s)) - (interp - 1) // 2
                o.append(b)
                ws.append(_lagrange(k, s - b))
            org.append(o)
            wt.append(ws)
        length = (5 if weno else k, k, k)
        lo = [int(min(float(b.min()) for b in org[a])) for a in range(3)]
        hi = [int(max(float(b.max()) for b in org[a])) + length[a] - 1 for a in range(3)]
        if max(-min(lo), max(hi)) > halo:
            raise RuntimeError("a departure point beyond the halo")
        zero = torch.zeros_like(T)

        def at(ax, i, o, weights):  # weight of offset o in the window of class i
            r = zero
            for j, v in enumerate(weights):
                r = torch.where(org[ax][i] + j == o, v, r)
            return r

        acc = [torch.zeros((q1, q1, q1) + n, dtype=f.dtype, device=f.device) for _ in srcs]
        S = [torch.zeros_like(acc[0]) for _ in range(3)] if weno else None
        row = [torch.zeros_like(acc[0]) for _ in range(5)] if weno else None
        for ox in range(lo[0], hi[0] + 1):
            for oy in range(lo[1], hi[1] + 1):
                wy = [at(1, i, oy, wt[1][i]) for i in range(q1)]
                for oz in range(lo[2], hi[2] + 1):
                    o = (ox, oy, oz)
                    wz = [at(2, i, oz, wt[2][i]) for i in range(q1)]
                    wx = None if weno else [at(0, i, ox, wt[0][i]) for i in range(q1)]
                    M = []
                    for ax in range(3):
                        s, r = (cut(us[ax], o) - U[ax]) / C, cut(cs[ax], o) / C
                        M.append([[_basis(q1, i, s + r * xi[b]) for b in range(q1)] for i in range(q1)])
                        if not weno:
                            v = (wx, wy, wz)[ax]
                            M[ax] = [[v[i] * t for t in M[ax][i]] for i in range(q1)]
                    for d, s in enumerate(srcs):
                        t = cut(s, o).reshape((q1, q1, q1) + n)
                        for ax in (2, 1, 0):
                            t = contract(M[ax], t, ax)
                        if not weno:
                            acc[d] += t
                            continue
                        for i1 in range(q1):
                            mid = torch.stack([torch.stack([((org[1][i2] + 1 == oy) & (org[2][i3] + 1 == oz))
                                                            for i3 in range(q1)]) for i2 in range(q1)])
                            wyz = torch.stack([torch.stack([wy[i2] * wz[i3] for i3 in range(q1)]) for i2 in range(q1)])
                            for j in range(3):
                                S[j][i1] += _at_shift(org[0][i1] + j, wt[0][i1][j], ox) * wyz * t[i1]
                            for m in range(5):
                                row[m][i1] += ((org[0][i1] + m == ox) & mid) * t[i1]
        if weno:
            for i1 in range(q1):
                acc[0][i1] = _weno_blend([v[i1] for v in S], [v[i1] for v in row], dist[i1])
        flat = [a.reshape((q1 ** 3,) + n) for a in acc]
        r = flat[0].sum(0)
        m = [torch.zeros_like(T) for _ in range(3)]
        e = torch.zeros_like(T)
        for t in range(q1 ** 3):
            cl = (t // (q1 * q1), t // q1 % q1, t % q1)
            v = [C * xi[cl[a]] + U[a] for a in range(3)]
            for a in range(3):
                m[a] += flat[0][t] * v[a]
            e += flat[0][t] * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
        if h is not None:
            e = flat[1].sum(0)
        m = torch.stack([a / r for a in m])
        return (flat[0], flat[-1], r), m, (e / r - (m * m).sum(0)) / (3 + dof)

    (fa, ha, r), U, T = _converge(evaluate, U, T)
    beta = 1.0 / case["tau"]
    fo, ho, C = torch.empty_like(f), torch.empty_like(f) if h is not None else None, torch.sqrt(T / tlat)
    for t, q in enumerate(order):
        fo[q] = fa[t] + beta * (r * w[t] - fa[t])
        if h is not None:
            cl = (t // (q1 * q1), t // q1 % q1, t % q1)
            v2 = sum((C * xi[cl[a]] + U[a]) ** 2 for a in range(3))
            ho[q] = ha[t] + beta * (r * w[t] * (v2 + dof * T) - ha[t])
    out = (fo, r, torch.cat([U, T[None]]))
    return out if h is None else out + (ho,)


def _at_shift(start, weights, o):
    """sum over the three nodes from `start` of the weight that sits at offset o"""
    r = torch.zeros_like(start)
    for j, v in enumerate(weights):
        r = torch.where(start + j == o, v, r)
    return r


def _exact1d(case, f, rho, g, first=None, last=None, mask=None):
    """One D1Q5 step: f [5, N], g [2, N] = u, T in float64; stencils held between first and last (clamp),
    or on a periodic grid with a node mask."""
    xi, w, interp, n = XI[5], W1[5], case["interp"], rho.numel()
    x = torch.arange(n, device=f.device)
    u0, T0 = g[0], g[1]
    c0 = torch.sqrt(T0)
    if mask is not None:
        # nearest active node at or before / after every position, as unwrapped indices
        pos = torch.cat([x, x + n])
        prev = torch.cummax(torch.where(torch.cat([mask, mask]), pos, torch.full_like(pos, -1)), 0).values[n:]
        nxt = torch.flip(torch.cummin(torch.flip(torch.where(torch.cat([mask, mask]), pos, torch.full_like(pos, 4 * n)),
                                                 [0]), 0).values, [0])[:n]
        back, ahead = x + n - prev, nxt - x  # distances to the active nodes

    def moved(k, idx, U, C):  # population k of the nodes idx [..., N] in the gauge (U, C)
        s, r = (u0[idx] - U) / C, c0[idx] / C
        return sum(_basis(5, k, s + r * xi[b]) * f[b][idx] for b in range(5))

    def evaluate(Ug, T):
        U, C = Ug[0], torch.sqrt(T)
        acc = []
        for k in range(5):
            v = C * xi[k] + U
            if mask is not None:
                s = x - v
                fl = torch.floor(s)
                i = (fl.long() % n)
                l, dl = (i - back[i]) % n, back[i]
                j = (i + 1) % n
                r, dr = (j + ahead[j]) % n, ahead[j]
                sl, sr = s - fl + dl, fl + 1 - s + dr
                acc.append((sr * moved(k, l, U, C) + sl * moved(k, r, U, C)) / (sl + sr))
                continue
            hold = lambda i: torch.minimum(torch.maximum(i, first), last)  # noqa: E731
            if interp == TVD:
                F = []
                for m in (-2.0, -1.0, 0.0, 1.0):
                    s = m * v
                    b = torch.floor(s) - 1
                    ws = _lagrange(4, s - b)
                    F.append(sum(ws[j] * moved(k, hold(x + b.long() + j), U, C) for j in range(4)))

                def minmod(a, b):
                    return torch.where(a * b <= 0, torch.zeros_like(a), torch.where(a.abs() < b.abs(), a, b))

                sg = torch.sign(v)
                d = F[2] - F[1]
                acc.append(F[2] - (d + 0.5 * sg * minmod(d, F[3] - F[2]) - 0.5 * sg * minmod(d, F[1] - F[0])))
            else:
                s = -v
                m = torch.floor(s + 0.5)
                p = [moved(k, hold(x + m.long() + j - 2), U, C) for j in range(5)]
                S = []
                for j in range(3):
                    ws = _lagrange(3, s - (m - 2 + j))
                    S.append(sum(a * b for a, b in zip(ws, p[j:j + 3])))
                acc.append(_weno_blend(S, p, s - m))
        acc = torch.stack(acc)
        r = acc.sum(0)
        m1 = sum(acc[k] * (C * xi[k] + U) for k in range(5)) / r
        m2 = sum(acc[k] * (C * xi[k] + U) ** 2 for k in range(5)) / r
        Tn = m2 - m1 * m1
        if mask is not None:
            m1, Tn = torch.where(mask, m1, u0), torch.where(mask, Tn, T0)
            acc, r = torch.where(mask, acc, f), torch.where(mask, r, rho)
        return (acc, r), m1[None], Tn

    (fa, r), U, T = _converge(evaluate, u0[None], T0)
    weights = torch.tensor(w, dtype=f.dtype, device=f.device)[:, None]
    fo = fa + (r * weights - fa) / case["tau"]
    if mask is not None:
        fo = torch.where(mask, fo, f)
    return fo, r, torch.stack([U[0], T])


def exact(case, seed):
    path = case["path"]
    if path == "batch":
        lengths, rho, u, T = _tubes(case, seed)
        if rho.size * case["steps"] > 6_000_000:
            return None
        dev = torch.device("cuda")
        r, u, T = (torch.from_numpy(a.astype(np.float32)).to(dev).double() for a in (rho, u, T))
        f = (torch.from_numpy(rho).to(dev) * torch.tensor(W1[5], dtype=torch.float64, device=dev)[:, None])
        f, g = f.float().double(), torch.stack([u, T])
        end = torch.from_numpy(np.repeat(np.cumsum(lengths, dtype=np.int64), lengths)).to(dev) - 1
        start = torch.from_numpy(np.repeat(np.cumsum(lengths, dtype=np.int64) - lengths, lengths)).to(dev)
        for _ in range(case["steps"]):
            f, r, g = _exact1d(case, f, r, g, start, end)
        return f.cpu().numpy(), r.cpu().numpy(), g[0].cpu().numpy(), g[1].cpu().numpy()
    n, q1 = (case["nz"], case["ny"], case["nx"]), _lattice(case)[0]
    if path == "host":
        if n[0] * n[1] * n[2] > 1_000_000:
            return None
        out = []
        for k in range(3):
            f, rho, g = (t.double() for t in _state(_host_case(case), seed * 3 + k))
            f, rho, g = _exact3d(_host_case(case), f.reshape((-1,) + n), rho.reshape(n), g.reshape((4,) + n))
            out.append((rho.reshape(-1).cpu(), g.reshape(4, -1).cpu()))
        return out
    if path in ("d1q5", "mesh"):
        f, rho, g = (t.double() for t in _state(case, seed))
        g = torch.stack([g[0], g[3]])
        x = torch.arange(rho.numel(), device=rho.device)
        ends = (torch.zeros_like(x), torch.full_like(x, rho.numel() - 1))
        for _ in range(case["steps"]):
            f, rho, g = _exact1d(case, f, rho, g, *ends, mask=_mask(case, seed) if path == "mesh" else None)
        zero = torch.zeros_like(rho)
        return f, rho, torch.stack([g[0], zero, zero, g[1]])
    if n[0] * n[1] * n[2] * q1 ** 3 * case["steps"] > 120_000_000:
        return None
    f, rho, g = (t.double() for t in _state(case, seed))
    f, rho, g = f.reshape((-1,) + n), rho.reshape(n), g.reshape((4,) + n)
    if path == "energy":
        dof, order, w, xi = 2, ORDER27, _weights(3, 3), XI[3]
        C, h = torch.sqrt(g[3] * 3), torch.empty_like(f)
        for t, q in enumerate(order):
            v2 = sum((C * xi[c] + g[a]) ** 2 for a, c in enumerate((t // 9, t // 3 % 3, t % 3)))
            h[q] = (rho * w[t] * (v2 + dof * g[3])).float().double()
        for _ in range(case["steps"]):
            f, rho, g, h = _exact3d(case, f, rho, g, h, dof)
    else:
        for _ in range(case["steps"]):
            f, rho, g = _exact3d(case, f, rho, g)
    return f.reshape(f.shape[0], -1), rho.reshape(-1), g.reshape(4, -1)
