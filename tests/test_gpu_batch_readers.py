"""Several threads read the same batch back at once: every one gets the batch's state."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("problems", [20, 120])
def test_readers_do_not_share_buffers(pond, problems):
    """Below and above the size from which the read-back goes through the batch's pinned buffers."""
    from lbmpond_b200.batch import Batch
    rng = np.random.default_rng(problems)
    lengths = np.full(problems, 3001)
    n = int(lengths.sum())
    assert (n > 200000) == (problems == 120)
    rho, u, T = (rng.uniform(0.5, 1.5, n).astype(np.float32).astype(float) for _ in range(3))
    wrong = []

    def reader(b):
        for _ in range(10):
            _, r, uu, tt = b.get_state()
            if not (np.array_equal(r, rho) and np.array_equal(uu, u) and np.array_equal(tt, T)):
                wrong.append(1)

    with Batch(lengths) as b:
        b.set_state(rho, u, T)
        threads = [threading.Thread(target=reader, args=(b,)) for _ in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not wrong
