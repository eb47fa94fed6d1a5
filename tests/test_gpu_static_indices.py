"""swb_sweep_static takes the lcg32 parameter indices from the caller's device memory: a byte past the last
pair acts as the last pair."""
import numpy as np
import pytest

from oracle import num_tiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L0,L1,tile,W", [(64, 48, (16, 8), 16), (62, 50, (32, 6), 8), (96, 64, (8, 5), 32)])
def test_indices_past_the_last_pair(gpu, oracle, L0, L1, tile, W):
    import torch
    nt = num_tiles(L0, L1, *tile)
    rng = oracle.rng_init(W, nt, 3)
    sel = np.random.default_rng(1).integers(0, 5, nt * W).astype(np.uint8)
    past = np.where(sel == 4, np.resize(np.array([4, 5, 130, 255], np.uint8), nt * W), sel).astype(np.uint8)
    got = []
    for s in (sel, past):
        bufs = [torch.from_numpy(x).cuda() for x in (oracle.hot_start(L0, L1, 2).reshape(-1).copy(),
                                                     rng.state.reshape(-1).view(np.int32).copy(), s.copy(),
                                                     rng.iteration.view(np.int32).copy())]
        torch.cuda.synchronize()
        assert gpu.lib().swb_sweep_static(None, L0, L1, tile[0], tile[1], W, 2.2691853, 3,
                                          *(b.data_ptr() for b in bufs), 1) == 0
        got.append([b.cpu().numpy() for b in bufs])
    for a, b in zip(*got):
        assert np.array_equal(a, b)
