"""Steps whose kernels start while the step before still runs (launch_early in
pond_step.cu)."""
import os
import re

import numpy as np
import pytest

from tests.states import perturbed_populations, smooth_state

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lbmpond_b200", "csrc")


@pytest.mark.parametrize("name", ["pond_step_1d_warp.cuh", "pond_step_d3q27.cuh"])
def test_overlapped_kernels_use_plain_loads(name):
    """Their inputs are written while they are resident, which the read-only path does not allow: neither
    __ldg nor the helpers that use it (load_node, transfer_one_1d, MeshNode)."""
    code = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    assert "cudaGridDependencySynchronize()" in code
    assert not re.search(r"__ldg|ld\.global\.nc|load_node\s*<|transfer_one_1d|MeshNode", code)
    # the kernels that take a programmatic launch are in these files
    launches = re.findall(r"= ?launch_early\(&?([\w:]+)|return launch_early\(&?([\w:]+)",
                          open(os.path.join(CSRC, "pond_step.cu")).read())
    assert sorted(a or b for a, b in launches) == ["d27::pull_d3q27_tile_kernel", "kern"]


@pytest.mark.gpu
@pytest.mark.parametrize("lattice,shape,interp,precision,bc", [
    (0, (900, 1, 1), 7, "fp64", (1, 0, 0)), (0, (3001, 1, 1), 8, "fp32", (2, 0, 0)), (0, (257, 1, 1), 4, "fp32", (0, 0, 0)),
    (1, (21, 13, 9), 4, "fp32", (2, 1, 0)), (1, (45, 18, 10), 3, "fp32", (2, 2, 1)), (1, (24, 24, 24), 2, "fp32", (0, 0, 0))])
def test_overlapped_steps_equal_single_steps(orc, pond, lattice, shape, interp, precision, bc):
    dim = 1 if lattice == 0 else 3
    rho, g = smooth_state(shape, dim, seed=5, modes=1, T0=0.02 if dim == 1 else 0.08, du=0.02, dT=0.002)
    f = perturbed_populations(orc, lattice, rho, g, seed=5, eps=0.01)
    states = []
    for calls in ((12,), (1,) * 12):
        with pond.Solver(lattice=lattice, shape=shape, interp=interp, precision=precision, tau=0.8, bc=bc) as s:
            s.set_state(rho, g, f=f)
            for n in calls:
                s.step(n)
                s.diagnostics()
            states.append(s.get_state())
    for a, b in zip(*states):
        assert np.array_equal(a, b)
