"""pond_step_noalloc forms its sums in a fixed order on every grid it accepts:
repeating a step repeats them to the last bit."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,interp", [((1024, 2728, 6), 4), ((2048, 4096, 2), 2), ((256, 256, 64), 3)])
def test_sums_repeat_bit_for_bit(pond, shape, interp):
    """The first two have 174,592 and 262,144 tiles for 65,536 records."""
    import torch
    from lbmpond_b200 import _lib
    from tests.test_zz_no_alloc import _bind
    L = _lib.load()
    N = int(np.prod(shape))
    p = _lib.PondParams()
    assert L.pond_params_default(1, ctypes.byref(p)) == 0
    p.Nx, p.Ny, p.Nz = shape
    p.interp, p.tau, p.max_iter = interp, 0.8, 2
    gen = torch.Generator("cuda").manual_seed(interp)

    def noise(*n):
        return torch.rand(n, generator=gen, device="cuda") * 2 - 1

    rho = 1 + 0.1 * noise(N)
    g = torch.cat([0.02 * noise(3, N), 0.05 * (1 + 0.1 * noise(1, N))])
    f = torch.as_tensor(pond.lattice_tables(1)[1], dtype=torch.float32, device="cuda")[:, None] * rho
    out = [torch.empty_like(t) for t in (f, rho, g)]
    seen = []
    for _ in range(4):
        diag = torch.zeros(ctypes.sizeof(_lib.PondDiag), dtype=torch.uint8, device="cuda")
        st = _bind(L)(ctypes.byref(p), f.data_ptr(), rho.data_ptr(), g.data_ptr(), *(t.data_ptr() for t in out),
                      diag.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert st == 0, L.pond_last_error_string().decode()
        torch.cuda.synchronize()
        seen.append(bytes(diag.cpu().numpy()))
    d = _lib.PondDiag.from_buffer_copy(seen[0])
    # 2 N + .. float64 additions in trees and runs of at most 1,100: far below 1e-12
    assert abs(d.mass - out[1].double().sum().item()) <= 1e-12 * d.mass
    assert d.niter_max == 2 and N < d.niter_sum <= 2 * N
    assert all(s == seen[0] for s in seen)
