"""The one-kernel sweep of lattices that fit one thread-block cluster (csrc/sw_whole.cuh): one CTA and
clusters of 2 to 16, CTAs without rows at the end, a single strip (its last column next to its first),
partial strips, rows and tiles, tiles of two and 32 rows, every tile width with every lcg width, 4-, 2- and
1-byte stores, lists that overflow, and samples taken by the next sweep; bit for bit against the
restatement and one launch a sweep."""
import numpy as np
import pytest

from oracle import num_tiles

pytestmark = pytest.mark.gpu

CASES = [
    # (L0, L1, tile, W, T, ordered start)
    (2, 2, (16, 8), 16, 2.2691853, False),
    (2, 64, (8, 2), 8, 2.0, False),
    (32, 32, (16, 8), 16, 2.2691853, False),    # one CTA, one strip
    (30, 18, (8, 5), 32, 2.3, False),
    (64, 64, (16, 4), 16, 2.0, False),
    (62, 130, (16, 8), 16, 2.2691853, False),   # 2-byte rows, partial tile row
    (128, 128, (16, 8), 16, 2.2691853, False),  # four CTAs
    (128, 72, (16, 8), 16, 2.5, False),         # nine tile rows: CTAs without rows
    (256, 256, (16, 8), 16, 2.2691853, False),  # 16 CTAs
    (512, 256, (16, 8), 16, 1.8, False),        # two bands of 16 strips a CTA
    (250, 258, (8, 8), 8, 2.2691853, False),
    (160, 512, (32, 32), 8, 2.3, False),
    (96, 66, (32, 3), 16, 3.0, False),
    (200, 100, (16, 16), 32, 2.2, False),
    (256, 192, (8, 8), 16, 0.05, True),         # one cluster winds around both ways
]


@pytest.mark.parametrize("L0,L1,tile,W,T,ordered", CASES)
def test_whole_sweeps_bit_exact_vs_oracle(gpu, oracle, L0, L1, tile, W, T, ordered):
    spins = oracle.hot_start(L0, L1, 2)
    if ordered:
        spins[...] = 1
        spins[L1 // 3:L1 // 3 + 9, ::2] = 0
    rng = oracle.rng_init(W, num_tiles(L0, L1, *tile), 3)
    with gpu.SwendsenWang2D(L0, L1, tile, W, 3) as sw:
        assert sw.launches_per_sweep() == 1
        sw.set_spins(spins)
        for n in (1, 7):
            sw.update(T, n)
            for _ in range(n):
                oracle.sweep(spins, tile[0], tile[1], rng, T=T)
            assert np.array_equal(sw.get_spins(), spins)
        st, a, c, it = sw.get_rng()
        assert np.array_equal(st, rng.state) and np.array_equal(it, rng.iteration)
        assert np.array_equal(a, rng.a) and np.array_equal(c, rng.c)
        # the phase kernels go on from there, and back
        assert np.array_equal(sw.update_dumped(T)[2], oracle.sweep(spins, tile[0], tile[1], rng, T=T, dumps=True)[2])
        sw.update(T, 1)
        oracle.sweep(spins, tile[0], tile[1], rng, T=T)
        assert np.array_equal(sw.get_spins(), spins)


@pytest.mark.parametrize("L0,L1", [(64, 48), (256, 256), (34, 50)])
def test_whole_samples(gpu, oracle, L0, L1):
    spins = oracle.hot_start(L0, L1, 1)
    rng = oracle.rng_init(16, num_tiles(L0, L1, 16, 8), 1)
    want = []
    with gpu.SwendsenWang2D(L0, L1, (16, 8), 16) as sw:
        sw.set_spins(spins)
        sw.update(2.3, 12, measure_every=3)
        for k in range(12):
            oracle.sweep(spins, 16, 8, rng, T=2.3)
            if (k + 1) % 3 == 0:
                want.append(oracle.energy_magnetization(spins))
        assert [tuple(x) for x in sw.samples()] == want


def test_whole_in_bands_and_combs(gpu, oracle):
    """Lists that overflow: every equal pair bonded, combs whose teeth the next row unites, 32-row tiles."""
    L0, L1, tile = 128, 64, (16, 32)
    y, x = np.mgrid[0:L1, 0:L0]
    spins = np.where(y % 3 == 0, x & 1, y % 3 == 1).astype(np.uint8)
    rng = oracle.rng_init(16, num_tiles(L0, L1, *tile), 1)
    with gpu.SwendsenWang2D(L0, L1, tile, 16) as sw:
        assert sw.launches_per_sweep() == 1
        sw.set_spins(spins)
        sw.update(0.05, 2)
        for _ in range(2):
            oracle.sweep(spins, *tile, rng, T=0.05)
        assert np.array_equal(sw.get_spins(), spins)
