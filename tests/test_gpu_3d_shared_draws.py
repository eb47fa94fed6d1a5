"""Small 3D lattices, whose blocks are made smaller where they would draw in more passes than a CTA has warps
(csrc/sw_3d.cuh, spread3) and whose warps take a piece's draws between them (csrc/sw_3d.cu, draw_share3): shares
that do and do not divide the passes, empty passes and pieces, whole and cut tiles, two row groups, and
lattices with more blocks than either rule asks for.  Bit for bit against the 3D restatement."""
import numpy as np
import pytest

from oracle import num_tiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L0,L1,L2,tile,W", [
    (42, 36, 2, (8, 1, 5), 32),      # 3 pieces of 24 passes, cut layers
    (96, 26, 2, (8, 2, 1), 32),      # 2 pieces of 32 passes
    (2, 14, 4, (8, 2, 2), 32),       # one tile column of four
    (90, 52, 26, (8, 1, 6), 32),     # 8 pieces
    (24, 30, 20, (8, 3, 3), 16),     # 10 pieces: no warp left over
    (34, 20, 16, (16, 8, 8), 32),    # 64 rows a piece
    (16, 16, 1, (16, 4, 1), 8),
    (64, 8, 6, (32, 2, 6), 16),
    (38, 12, 60, (8, 1, 3), 32),     # 8 blocks become 64
    (2, 48, 36, (16, 4, 1), 32),
    (128, 96, 64, (32, 1, 1), 8),    # 96 blocks of 16 one-row pieces
    (160, 80, 64, (8, 1, 1), 32),    # 64 passes a piece
    (32, 32, 16 * 148, (16, 4, 4), 16),  # 296 blocks: not shared
    (32, 32, 16 * 74, (16, 4, 4), 16),   # 148 blocks: shared
])
def test_shared_draws_bit_exact(gpu, oracle, L0, L1, L2, tile, W):
    spins = np.random.default_rng(L0 + L1 + L2).integers(0, 2, (L2, L1, L0), dtype=np.uint8)
    r = oracle.rng_init(W, num_tiles(L0, L1, tile[0], tile[1]) * -(-L2 // tile[2]), 9)
    with gpu.SwendsenWang3D(L0, L1, L2, tile, W, 9) as sw:
        sw.set_spins(spins)
        sw.update(4.5115, 3)
        for _ in range(3):
            oracle.sweep3(spins, tile, r, T=4.5115)
        bonds, lab = oracle.sweep3(spins, tile, r, T=4.5115, dumps=True)
        gb, gl = sw.update_dumped(4.5115)
        assert np.array_equal(gb, bonds) and np.array_equal(gl, lab)
        assert np.array_equal(sw.get_spins(), spins)
        st, a, c, it = sw.get_rng()
        assert np.array_equal(st, r.state) and np.array_equal(it, r.iteration)
        assert np.array_equal(a, r.a) and np.array_equal(c, r.c)
