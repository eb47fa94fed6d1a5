"""The assign's label rows (csrc/sw_strip.cuh): blocks of one, two, three and four strips, rows of whole
quads and rows that end in half a quad, last blocks of every width class, one band and several.  Bonds,
block labels and resolved labels bit for bit against the restatement."""
import numpy as np
import pytest

from oracle import num_tiles

pytestmark = pytest.mark.gpu

T = 2.2691853


@pytest.mark.parametrize("L0,L1,tile,W", [
    (2, 34, (8, 4), 16), (16, 40, (16, 8), 16), (26, 66, (8, 6), 8), (28, 70, (16, 9), 32), (32, 64, (8, 8), 16),
    (54, 64, (8, 5), 16), (64, 96, (16, 4), 16), (60, 38, (32, 7), 8),              # two strips
    (98, 66, (16, 8), 16), (130, 64, (16, 8), 16), (194, 70, (8, 8), 32), (256, 62, (16, 3), 8),
    (30, 14300, (16, 8), 16), (64, 14400, (32, 16), 16), (514, 2900, (8, 8), 16),   # one band
])
def test_label_rows(gpu, oracle, L0, L1, tile, W):
    spins = oracle.hot_start(L0, L1, 8)
    rng = oracle.rng_init(W, num_tiles(L0, L1, *tile), 2)
    with gpu.SwendsenWang2D(L0, L1, tile, W, 2) as sw:
        geo = sw.geometry()
        sw.set_spins(spins)
        for _ in range(2):
            bonds, _, lf = oracle.sweep(spins, *tile, rng, T=T, dumps=True)
            gb, glb, glf = sw.update_dumped(T)
            assert np.array_equal(gb, bonds) and np.array_equal(glf, lf)
            assert np.array_equal(glb, oracle.block_labels(bonds, geo["block_x"], geo["block_y"]))
            assert np.array_equal(sw.get_spins(), spins)


@pytest.mark.parametrize("block", [(1, 0), (2, 0), (3, 2), (5, 1), (6, 0), (7, 4)])
@pytest.mark.parametrize("many", [False, True])
def test_label_rows_in_a_batch(gpu, oracle, block, many):
    """Block widths of 8 to 112 columns; with `many` at least 400 items, one band."""
    shapes = [(90, 64, (8, 8)), (112, 40, (16, 4)), (58, 66, (16, 8))] + ([(510, 512, (8, 4))] if many else [])
    state = []
    with gpu.BatchedSW(capacity=12) as b:
        for k, (L0, L1, tile) in enumerate(shapes * (3 if many else 1)):
            i = b.add(L0, L1, T, k + 1, tile, block)
            spins = oracle.hot_start(L0, L1, k + 1)
            b.set_spins(i, spins)
            state.append((i, tile, spins, oracle.rng_init(16, num_tiles(L0, L1, *tile), k + 1)))
        b.sweep(2)
        for i, tile, spins, rng in state:
            for _ in range(2):
                oracle.sweep(spins, *tile, rng, T=T)
            assert np.array_equal(b.get_spins(i), spins)


@pytest.mark.parametrize("L0,L1,tile,W", [(2, 65600, (16, 8), 16), (30, 66000, (8, 8), 8), (64, 66000, (32, 16), 32)])
def test_narrow_lattices_of_many_blocks(gpu, oracle, L0, L1, tile, W):
    """More than 2048 blocks of one or two strips: sweeps and samples one after the other."""
    spins = oracle.hot_start(L0, L1, 4)
    rng = oracle.rng_init(W, num_tiles(L0, L1, *tile), 6)
    want = []
    with gpu.SwendsenWang2D(L0, L1, tile, W, 6) as sw:
        geo = sw.geometry()
        assert geo["blocks_x"] * geo["blocks_y"] > 2048
        sw.set_spins(spins)
        sw.update(T, 4, measure_every=2)
        for k in range(4):
            oracle.sweep(spins, *tile, rng, T=T)
            if k % 2:
                want.append(oracle.energy_magnetization(spins))
        assert [tuple(s) for s in sw.samples()] == want
        assert np.array_equal(sw.get_spins(), spins)
        st, a, c, it = sw.get_rng()
        assert np.array_equal(st, rng.state) and np.array_equal(it, rng.iteration)
