"""Sweeps in one kernel followed directly by sweeps in phase kernels and back, with nothing on the stream
or the host between them that waits: the assign must not draw from streams that the one-kernel sweep
still writes.  Spins and lcg32 streams bit for bit against the restatement."""
import numpy as np
import pytest

from oracle import num_tiles

pytestmark = pytest.mark.gpu

T = 2.2691853


@pytest.mark.parametrize("L0,L1,tile,W", [(32, 32, (16, 8), 16), (128, 128, (16, 8), 16), (256, 256, (8, 4), 32),
                                          (512, 256, (16, 8), 16), (250, 258, (8, 8), 8)])
@pytest.mark.parametrize("timed", [False, True])
def test_phase_kernels_right_after_one_kernel_sweeps(gpu, oracle, L0, L1, tile, W, timed):
    spins = oracle.hot_start(L0, L1, 3)
    rng = oracle.rng_init(W, num_tiles(L0, L1, *tile), 7)
    with gpu.SwendsenWang2D(L0, L1, tile, W, 7) as sw:
        assert sw.launches_per_sweep() == 1
        sw.set_spins(spins)
        n = 0
        for k in range(1, 9):
            sw.update(T, k)
            if timed:
                sw.sweep_timed(T, 2, per_kernel=True)
                n += k + 2
            else:
                assert gpu.lib().swb_sweep_dumped(sw._h, T, None, None, None) == 0
                n += k + 1
        for _ in range(n):
            oracle.sweep(spins, *tile, rng, T=T)
        assert np.array_equal(sw.get_spins(), spins)
        st, a, c, it = sw.get_rng()
        assert np.array_equal(st, rng.state) and np.array_equal(it, rng.iteration)
        assert np.array_equal(a, rng.a) and np.array_equal(c, rng.c)
