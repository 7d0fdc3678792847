"""The batched 1D kernel's two ways through an iteration (windows near each
other, or anywhere), the bin choice of small batches, and the threaded
read-back.  Tolerance as in test_gpu_batch.py: 3e-5 of the largest value of a
problem's field after a few steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WENO5, LAGR4 = 8, 4
LENGTHS = [3, 40, 700, 1201, 256, 2000, 1500, 512]


def _problems(lengths, seed):
    """Cold tubes (c about 0.3), every third with a hot stretch: wider than an eighth of the problem (the
    general way) in the even ones, narrower (single nodes take it) in the odd ones."""
    rng = np.random.default_rng(seed)
    rho, u, T = [], [], []
    for p, n in enumerate(lengths):
        x = np.arange(n)
        s = 0.5 * (1 + np.tanh((x - n / 2) / 4.0))
        r, t, v = rng.uniform(0.6, 1.6, 2), rng.uniform(0.07, 0.11, 2), rng.uniform(-0.05, 0.05, 2)
        hot = np.zeros(n)
        if p % 3 == 2:
            half = n / 4 if p % 2 == 0 else n / 20
            hot = 0.5 * (np.tanh((x - n / 3 + half / 2) / 8.0) - np.tanh((x - n / 3 - half / 2) / 8.0))
        rho.append(r[0] + (r[1] - r[0]) * s)
        T.append(t[0] + (t[1] - t[0]) * s + 0.3 * hot)
        u.append(v[0] + (v[1] - v[0]) * s)
    return np.concatenate(rho), np.concatenate(u), np.concatenate(T)


@pytest.mark.parametrize("interp", [WENO5, LAGR4])
def test_both_ways_match_oracle(orc, pond, interp):
    from lbmpond_b200.batch import Batch
    rho, u, T = _problems(LENGTHS, seed=interp)
    with Batch(LENGTHS, interp=interp, tau=0.7) as b:
        b.set_state(rho, u, T)
        b.run(4, steps_per_launch=2)
        f, r, uu, tt = b.get_state()
        assert b.stats()["nonconverged"] == 0
    for p, n in enumerate(LENGTHS):
        sl = slice(int(np.sum(LENGTHS[:p])), int(np.sum(LENGTHS[:p + 1])))
        ref = orc.base_state(0, rho[sl], u[sl], 0.0, 0.0, T[sl])
        for _ in range(4):
            ref, _, nc = orc.step(ref, 0, (n, 1, 1), interp=interp, tau=0.7, bc=(1, 1, 1))
            assert nc == 0
        cs = np.sqrt(ref.g[3].max())
        for got, want, scale in ((r[sl], ref.rho, ref.rho.max()), (uu[sl], ref.g[0], cs), (tt[sl], ref.g[3], ref.g[3].max()),
                                 (f[:, sl], ref.f, np.abs(ref.f).max())):
            assert np.abs(got - want).max() <= 3e-5 * scale, p


def test_tiles_and_packings_agree_bit_for_bit(pond):
    """Every way through an iteration rounds alike: another lane cap (which moves iterations to the warp-wide
    phase), or the problem alone in its batch, changes nothing."""
    from lbmpond_b200.batch import Batch
    rho, u, T = _problems(LENGTHS, seed=1)

    def run(lengths, sel, tile=None):
        with Batch(lengths) as b:
            if tile:
                b.tile = tile
            b.set_state(rho[sel], u[sel], T[sel])
            b.run(3)
            return b.get_state()

    full = run(LENGTHS, slice(None))
    for cap in (1, 2, 100):
        for x, y in zip(full, run(LENGTHS, slice(None), (512, cap))):
            assert np.array_equal(x, y), cap
    p = 6
    sl = slice(int(np.sum(LENGTHS[:p])), int(np.sum(LENGTHS[:p + 1])))
    for x, y in zip(full, run(LENGTHS[p:p + 1], sl)):
        assert np.array_equal(x[..., sl], y)


@pytest.mark.parametrize("count", [3, 90])
def test_read_back_puts_every_node_in_its_place(pond, count):
    """Both read-backs (plain; chunked over threads above 200,000 nodes) on problems of uneven length."""
    from lbmpond_b200.batch import Batch
    rng = np.random.default_rng(count)
    lengths = rng.integers(1, 4097, count * 2)
    lengths[:count] = rng.integers(3000, 4097, count)
    n = int(lengths.sum())
    assert (n > 200000) == (count == 90)
    rho, u, T = (rng.uniform(0.5, 1.5, n).astype(np.float32).astype(float) for _ in range(3))
    with Batch(lengths) as b:
        b.set_state(rho, u, T)
        for _ in range(2):
            f, r, uu, tt = b.get_state()
            assert np.array_equal(r, rho) and np.array_equal(uu, u) and np.array_equal(tt, T)
            w = f[:, 0] / rho[0]
            assert np.abs(f - w[:, None] * rho).max() <= 1e-6
