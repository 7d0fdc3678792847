"""The batch kernel's ways and tile widths round alike: tubes whose nodes run to
the iteration cap would turn a last digit into percents within some hundred steps."""
import numpy as np
import pytest

from tests.test_gpu_batch_routes import LENGTHS, _problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("interp", [8, 4])
@pytest.mark.parametrize("steps", [3, 40])
def test_all_widths_agree_bit_for_bit(pond, interp, steps):
    from lbmpond_b200.batch import Batch
    rho, u, T = _problems(LENGTHS, seed=2)
    outs = []
    for tile in ((512, 8), (512, 1), (256, 3), (768, 4), (768, 100), (1024, 2), (1024, 100)):
        with Batch(LENGTHS, interp=interp) as b:
            b.tile = tile
            b.set_state(rho, u, T)
            b.run(steps)
            outs.append((tile, b.get_state()))
    for tile, out in outs[1:]:
        for x, y in zip(outs[0][1], out):
            assert np.array_equal(x, y), tile
