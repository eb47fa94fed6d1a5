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


def _check_streams(got, rng):
    st, a, c, it = got
    assert np.array_equal(st, rng.state) and np.array_equal(it, rng.iteration)
    assert np.array_equal(a, rng.a) and np.array_equal(c, rng.c)


@pytest.mark.parametrize("L0,L1,ty", [
    (32, 102, 17),    # one strip, whole tile rows
    (30, 94, 24),     # 2-byte rows, a short last tile
    (32, 8840, 17),   # 520 tile rows: no cluster holds the lattice, plain sweeps run the phase kernels
])
def test_2d_odd_ballots(gpu, oracle, L0, L1, ty):
    spins = oracle.hot_start(L0, L1, 6)
    rng = oracle.rng_init(8, num_tiles(L0, L1, 32, ty), 2)
    with gpu.SwendsenWang2D(L0, L1, (32, ty), 8, 2) as sw:
        assert sw.launches_per_sweep() == (3 if L1 > 8000 else 1)
        sw.set_spins(spins)
        sw.update(2.2691853, 2)
        for _ in range(2):
            oracle.sweep(spins, 32, ty, rng, T=2.2691853)
        bonds, _, lf = oracle.sweep(spins, 32, ty, rng, T=2.2691853, dumps=True)
        gb, _, glf = sw.update_dumped(2.2691853)
        assert np.array_equal(gb, bonds) and np.array_equal(glf, lf)
        assert np.array_equal(sw.get_spins(), spins)
        _check_streams(sw.get_rng(), rng)


@pytest.mark.parametrize("L0,L1,ty", [(32, 102, 17), (30, 94, 24)])
def test_2d_odd_ballots_static(gpu, oracle, L0, L1, ty):
    import torch
    pairs = [(1372383749, 1289706101), (2891336453, 1640531513), (2024337845, 797082193), (32310901, 626627237),
             (29943829, 1013904223)]
    spins = oracle.hot_start(L0, L1, 6)
    rng = oracle.rng_init(8, num_tiles(L0, L1, 32, ty), 2)
    sel = np.array([pairs.index((int(a), int(c))) for a, c in zip(rng.a.ravel(), rng.c.ravel())], np.uint8)
    d_spins = torch.from_numpy(spins.reshape(-1).copy()).cuda()
    d_state = torch.from_numpy(rng.state.reshape(-1).view(np.int32).copy()).cuda()
    d_sel, d_it = torch.from_numpy(sel).cuda(), torch.from_numpy(rng.iteration.view(np.int32).copy()).cuda()
    torch.cuda.synchronize()
    assert gpu.lib().swb_sweep_static(None, L0, L1, 32, ty, 8, 2.2691853, 3, d_spins.data_ptr(), d_state.data_ptr(),
                                      d_sel.data_ptr(), d_it.data_ptr(), 1) == 0
    for _ in range(3):
        oracle.sweep(spins, 32, ty, rng, T=2.2691853)
    assert np.array_equal(d_spins.cpu().numpy(), spins.reshape(-1))
    assert np.array_equal(d_state.cpu().numpy().view(np.uint32), rng.state.reshape(-1))
    assert np.array_equal(d_it.cpu().numpy().view(np.uint32), rng.iteration)


@pytest.mark.parametrize("block", [(1, 1), (3, 1)])
def test_2d_odd_ballots_in_a_batch_of_one_band(gpu, oracle, block):
    """At least 400 block items (the assign takes them in one band), one and three strips a block."""
    shapes = [(96, 3400, 17), (94, 2400, 24), (32, 3400, 17), (96, 1700, 17)]
    state = []
    with gpu.BatchedSW(capacity=4, lcg_width=8) as b:
        for k, (L0, L1, ty) in enumerate(shapes):
            i = b.add(L0, L1, 2.2691853, 10 * k + 1, (32, ty), block)
            spins = oracle.hot_start(L0, L1, k + 1)
            b.set_spins(i, spins)
            state.append((i, ty, spins, oracle.rng_init(8, num_tiles(L0, L1, 32, ty), 10 * k + 1)))
        assert sum(b.info(s[0])["blocks"] for s in state) >= 400
        b.sweep(2)
        for i, ty, spins, rng in state:
            for _ in range(2):
                oracle.sweep(spins, 32, ty, rng, T=2.2691853)
            assert np.array_equal(b.get_spins(i), spins)
            _check_streams(b.get_rng(i), rng)
