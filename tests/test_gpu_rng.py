"""The lcg32 throughput kernel (swb_lcg32_benchmark, the counterpart of TestRNG --target)
against the oracle's restatement of LCG32<CPU>::NextReal: the reported stream's last 64
numbers bit for bit, and the XOR of every number of every stream."""
import numpy as np
import pytest

from computational_physics_b200 import rng_bench


@pytest.mark.gpu
@pytest.mark.parametrize("W", [8, 16, 32])
def test_lcg32_kernel_matches_oracle(gpu, oracle, W):
    n_streams, per = 37, 64 // W
    updates = 45 * per          # crosses many parameter rotations (every 15th update)
    r = rng_bench.generate(n_streams, updates, lcg_width=W, seed_base=1, report_id=5)
    want_x = 0
    for s in range(n_streams):
        nums = oracle.next_real(W, 1 + s, [64] * (updates * W // 64))
        want_x ^= int(np.bitwise_xor.reduce(nums.view(np.uint32)))
        if s == 5:
            np.testing.assert_array_equal(r["report"].view(np.uint32), nums[-64:].view(np.uint32))
    assert r["checksum"] == want_x
    assert r["numbers"] == n_streams * updates * W and r["ms"] > 0


@pytest.mark.gpu
def test_lcg32_argument_errors(gpu):
    with pytest.raises(gpu.NativeError):
        rng_bench.generate(4, 3, lcg_width=16)        # not a multiple of 64 / 16
    with pytest.raises(gpu.NativeError):
        rng_bench.generate(4, 4, lcg_width=12)
    with pytest.raises(gpu.NativeError):
        rng_bench.generate(4, 4, lcg_width=16, report_id=4)


def _checksum_and_report(oracle, W, n_streams, updates, seed, report_id):
    x, report = 0, None
    for s in range(n_streams):
        nums = oracle.next_real(W, seed + s, [64] * (updates * W // 64))
        x ^= int(np.bitwise_xor.reduce(nums.view(np.uint32)))
        if s == report_id:
            report = nums[-64:].view(np.uint32)
    return x, report


@pytest.mark.gpu
@pytest.mark.parametrize("W", [8, 16, 32])
@pytest.mark.parametrize("n_streams,buffers", [(1, 1), (9, 2), (33, 3), (5, 4), (3, 15), (2, 16), (17, 31)])
def test_lcg32_kernel_edges(gpu, oracle, W, n_streams, buffers):
    """Update counts around the groups of 15 (none, one, remainders; `buffers` times 64 / W updates),
    stream counts that do not fill a warp or a CTA, and calls from two threads at once: equal to the
    oracle bit for bit."""
    import threading
    updates = buffers * (64 // W)
    got = {}

    def call(k):
        got[k] = rng_bench.generate(n_streams, updates, lcg_width=W, seed_base=100 + k, report_id=n_streams - 1)
    threads = [threading.Thread(target=call, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in (0, 1):
        x, report = _checksum_and_report(oracle, W, n_streams, updates, 100 + k, n_streams - 1)
        assert got[k]["checksum"] == x
        np.testing.assert_array_equal(got[k]["report"].view(np.uint32), report)
