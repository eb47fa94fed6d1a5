"""The assign phase's strips and bands (csrc/sw_strip.cuh) where they can go wrong: partial strips, extents
that allow only 4- or 2-byte loads, tile heights that leave a short band or a partial tile row, every tile
width with every lcg width (one to four passes of draws per tile row), one band (at least 445 blocks) and
several, and more unions in a strip than its list holds.  Bonds, block labels, resolved labels, spins
and lcg32 streams bit for bit against the restatement."""
import numpy as np
import pytest

from oracle import num_tiles

pytestmark = pytest.mark.gpu


def _combs(L0, L1):
    """Rows 1010.., 1111.., 0000..: with every equal pair bonded (T -> 0) each comb's teeth are new labels
    that the next row unites, about 160 unions in a 32 x 32 strip (its list holds 128)."""
    y, x = np.mgrid[0:L1, 0:L0]
    return np.where(y % 3 == 0, x & 1, (y % 3 == 1)).astype(np.uint8)


CASES = [
    # (L0, L1, tile, W, T, combs)
    (34, 62, (8, 5), 8, 2.2691853, False),
    (130, 66, (16, 7), 16, 2.0, False),
    (1538, 34, (32, 3), 16, 2.5, False),
    (258, 1026, (8, 2), 32, 2.2691853, False),
    (100, 94, (32, 31), 32, 3.0, False),
    (200, 70, (16, 32), 8, 2.2691853, False),
    (66, 40, (32, 12), 8, 1.7, False),
    (104, 36, (16, 10), 32, 2.3, False),
    (4098, 640, (16, 8), 16, 2.2691853, False),    # one band, 2-byte rows, labels row by row
    (4100, 610, (8, 6), 8, 2.0, False),            # one band, 4-byte rows, last block 4 columns wide
    (4096, 640, (16, 8), 16, 0.05, True),          # one band, lists overflow
    (256, 96, (8, 8), 16, 0.05, True),             # bands
]


@pytest.mark.parametrize("L0,L1,tile,W,T,combs", CASES)
def test_strips_bit_exact_vs_oracle(gpu, oracle, L0, L1, tile, W, T, combs):
    spins = _combs(L0, L1) if combs else oracle.hot_start(L0, L1, 3)
    rng = oracle.rng_init(W, num_tiles(L0, L1, *tile), 5)
    with gpu.SwendsenWang2D(L0, L1, tile, W, 5) as sw:
        geo = sw.geometry()
        sw.set_spins(spins)
        for warm in ((0, 2) if combs else (2,)):
            for _ in range(warm):
                oracle.sweep(spins, tile[0], tile[1], rng, T=T)
            sw.update(T, warm)
            bonds, _, lf = oracle.sweep(spins, tile[0], tile[1], rng, T=T, dumps=True)
            gb, glb, glf = sw.update_dumped(T)
            assert np.array_equal(gb, bonds)
            assert np.array_equal(glb, oracle.block_labels(bonds, geo["block_x"], geo["block_y"]))
            assert np.array_equal(glf, lf)
            assert np.array_equal(sw.get_spins(), spins)
        st, a, c, it = sw.get_rng()
        assert np.array_equal(st, rng.state) and np.array_equal(it, rng.iteration)
        assert np.array_equal(a, rng.a) and np.array_equal(c, rng.c)


@pytest.mark.parametrize("block", [(0, 0), (3, 1), (1, 2), (5, 3)])
@pytest.mark.parametrize("W", [8, 16, 32])
def test_batched_strips_bit_exact_vs_oracle(gpu, oracle, W, block):
    """Block shapes that are no power of two (strips with idle columns), all tile widths together."""
    shapes = [(96, 64, (8, 5)), (130, 34, (16, 8)), (62, 80, (32, 6)), (256, 128, (16, 4))]
    state = []
    with gpu.BatchedSW(capacity=8, lcg_width=W) as b:
        for k, (L0, L1, tile) in enumerate(shapes):
            i = b.add(L0, L1, 2.2691853, 10 * k + 1, tile, block)
            spins = oracle.hot_start(L0, L1, k + 1)
            b.set_spins(i, spins)
            state.append((i, tile, spins, oracle.rng_init(W, num_tiles(L0, L1, *tile), 10 * k + 1)))
        b.sweep(3)
        for i, tile, spins, rng in state:
            for _ in range(3):
                oracle.sweep(spins, tile[0], tile[1], rng, T=2.2691853)
            assert np.array_equal(b.get_spins(i), spins)
            st, a, c, it = b.get_rng(i)
            assert np.array_equal(st, rng.state) and np.array_equal(it, rng.iteration) and np.array_equal(a, rng.a)


@pytest.mark.parametrize("L1", [2016, 2048])
def test_batched_rounds_in_one_and_two_groups(gpu, oracle, L1):
    """2290 and 2338 block items, either side of the line between rounds launched directly as one group and
    rounds of two groups side by side; budgets that end in different rounds."""
    shapes = [(2048, 2048, 5), (2048, L1, 3), (1024, 1024, 4), (96, 64, 2)]
    if L1 == 2048:
        shapes.append((512, 256, 5))
    with gpu.BatchedSW(capacity=8) as b:
        ids = []
        for k, (L0, M, sweeps) in enumerate(shapes):
            ids.append(b.add(L0, M, 2.2691853, k + 1, (16, 8)))
            b.hot_start(ids[-1], k + 1)
            b.set_schedule(ids[-1], sweeps, 2)
        b.sweep(6, measure=True)
        for k, (i, (L0, M, sweeps)) in enumerate(zip(ids, shapes)):
            with gpu.SwendsenWang2D(L0, M, (16, 8), 16, k + 1) as sw:
                sw.hot_start(k + 1)
                sw.update(2.2691853, sweeps, 2)
                assert b.status(i) == (0, sweeps)
                assert np.array_equal(b.get_spins(i), sw.get_spins())
                assert np.array_equal(b.samples(i), sw.samples())
