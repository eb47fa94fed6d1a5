"""The 3D assign's pieces (csrc/sw_3d.cu) where they can go wrong: tile shapes whose face requests start
inside an update, tiles of more than 32 rows (two row groups), one-row tiles (many pieces), partial
blocks, pieces and tiles in every direction, every lcg width with every tile width, 2- and 4-byte rows,
more linked labels than a piece remembers; and measurements taken by the next sweep's assign phase.  Bit
for bit against the 3D restatement."""
import numpy as np
import pytest

from oracle import num_tiles

pytestmark = pytest.mark.gpu

CASES = [
    # (L0, L1, L2, tile, W, T)
    (40, 26, 22, (8, 5, 7), 16, 4.5115),     # 35 rows a tile: two groups
    (66, 34, 18, (16, 8, 8), 32, 4.0),       # 64 rows, partial everywhere, 2-byte rows
    (36, 20, 40, (8, 3, 3), 32, 5.0),        # face elements start inside an update
    (64, 40, 36, (32, 1, 1), 8, 4.5115),     # one-row tiles: 16 pieces of 16 rows
    (24, 48, 34, (8, 1, 8), 8, 4.5115),      # 24 columns: three tiles of a strip
    (100, 30, 12, (32, 7, 2), 16, 3.5),
    (16, 64, 2, (16, 2, 3), 16, 4.5),
    (34, 4, 130, (16, 6, 1), 8, 4.2),
]


def _run(gpu, oracle, spins, L0, L1, L2, tile, W, T, sweeps=3):
    nt = num_tiles(L0, L1, tile[0], tile[1]) * -(-L2 // tile[2])
    r = oracle.rng_init(W, nt, 9)
    with gpu.SwendsenWang3D(L0, L1, L2, tile, W, 9) as sw:
        sw.set_spins(spins)
        for _ in range(sweeps - 1):
            oracle.sweep3(spins, tile, r, T=T)
        sw.update(T, sweeps - 1)
        bonds, lab = oracle.sweep3(spins, tile, r, T=T, dumps=True)
        gb, gl = sw.update_dumped(T)
        assert np.array_equal(gb, bonds)
        assert np.array_equal(gl, lab)
        assert np.array_equal(sw.get_spins(), spins)
        st, a, c, it = sw.get_rng()
        assert np.array_equal(st, r.state) and np.array_equal(it, r.iteration)
        assert np.array_equal(a, r.a) and np.array_equal(c, r.c)
        assert sw.energy_magnetization_sums() == oracle.energy_magnetization3(spins)


@pytest.mark.parametrize("L0,L1,L2,tile,W,T", CASES)
def test_pieces_bit_exact_vs_oracle(gpu, oracle, L0, L1, L2, tile, W, T):
    spins = np.random.default_rng(L0 + L1 + L2).integers(0, 2, (L2, L1, L0), dtype=np.uint8)
    _run(gpu, oracle, spins, L0, L1, L2, tile, W, T)


@pytest.mark.parametrize("L0", [64, 66])
def test_more_linked_labels_than_a_piece_remembers(gpu, oracle, L0):
    """Layers: checkerboard, ones, the other checkerboard, zeros, with every equal pair bonded (T -> 0):
    each checkerboard's sites are new labels that the next layer unites, and the join unites again."""
    z, y, x = np.mgrid[0:32, 0:32, 0:L0]
    spins = np.choose(z % 4, [(x + y) & 1, np.ones_like(x), 1 - ((x + y) & 1), np.zeros_like(x)]).astype(np.uint8)
    _run(gpu, oracle, spins, L0, 32, 32, (16, 4, 4), 16, 0.05, sweeps=1)


@pytest.mark.parametrize("every", [1, 4])
def test_samples_taken_by_the_next_sweep(gpu, oracle, every):
    """Samples between calls, before a change of the spins and at the end, in order."""
    L0, L1, L2, tile = 48, 20, 18, (16, 4, 4)
    nt = num_tiles(L0, L1, 16, 4) * -(-L2 // 4)
    want = []
    with gpu.SwendsenWang3D(L0, L1, L2, tile, 16, 3) as sw:
        sw.hot_start(1)
        spins = sw.get_spins()
        r = oracle.rng_init(16, nt, 3)
        for n in (8, 4):
            sw.update(4.5, n, measure_every=every)
            for k in range(n):
                oracle.sweep3(spins, tile, r, T=4.5)
                if (k + 1) % every == 0:
                    want.append(oracle.energy_magnetization3(spins))
        sw.set_spins(np.zeros_like(spins))
        samples, acc = sw.samples()
    assert [tuple(s) for s in samples] == want and acc[3] == len(want)
