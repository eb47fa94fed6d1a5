"""Sweeps of tile shapes whose ballots fill an odd number of words, where every area behind them in shared
memory has to be brought back to its alignment (test_layouts.py walks all shapes on the host).  Bit for
bit against the restatement."""
import numpy as np
import pytest

from oracle import num_tiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L0,L1,L2,tile,W", [
    (64, 64, 64, (32, 4, 5), 8),     # 243 ballots a piece, 12 pieces a block
    (64, 64, 64, (16, 6, 8), 16),    # 147, two row groups
    (66, 30, 26, (32, 7, 7), 32),    # 149, 2-byte rows
    (24, 28, 40, (8, 7, 8), 8),      # 175
    (32, 4, 34, (32, 8, 5), 16),     # one piece a tile layer, three a block
])
def test_3d_odd_ballots(gpu, oracle, L0, L1, L2, tile, W):
    spins = np.random.default_rng(L0 + L2).integers(0, 2, (L2, L1, L0), dtype=np.uint8)
    r = oracle.rng_init(W, num_tiles(L0, L1, tile[0], tile[1]) * -(-L2 // tile[2]), 4)
    with gpu.SwendsenWang3D(L0, L1, L2, tile, W, 4) as sw:
        sw.set_spins(spins)
        sw.update(4.5115, 2)
        for _ in range(2):
            oracle.sweep3(spins, tile, r, T=4.5115)
        bonds, lab = oracle.sweep3(spins, tile, r, T=4.5115, dumps=True)
        gb, gl = sw.update_dumped(4.5115)
        assert np.array_equal(gb, bonds) and np.array_equal(gl, lab)
        assert np.array_equal(sw.get_spins(), spins)
        st, a, c, it = sw.get_rng()
        assert np.array_equal(st, r.state) and np.array_equal(it, r.iteration)
        assert np.array_equal(a, r.a) and np.array_equal(c, r.c)
