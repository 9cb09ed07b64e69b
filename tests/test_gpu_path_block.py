"""The block-per-swath path sweep of the DBA round against the CPU oracle, bit
for bit: row and column counts at the edges of its chunks, rings, warps and
swaths, and more swaths than the GPU holds blocks (a swath that starts after
its left neighbour has finished finds all its input waiting)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

MODES = [(0, 0), (1, 0), (0, 1), (1, 1)]


@pytest.fixture(scope="module")
def env():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opendba_b200 import api, build
    build.build_library()
    return torch, api


def _signal(rng, L, dtype):
    return (np.repeat(rng.normal(0, 1, L // 9 + 1), 9)[:L] + rng.normal(0, 0.1, L)).astype(dtype)


def _ranges(env, centroid, members, os_, oe):
    torch, api = env
    ds = api.DeviceSeries.from_host(members)
    c = torch.from_numpy(np.ascontiguousarray(centroid)).cuda()
    return api.dba_round_ranges(c, ds, os_, oe).cpu().numpy()


# rows around a row pair, a chunk of 8 steps (16 rows), the 31-step fill, the
# feeder's 16 pairs, the edge ring (128 pairs) and the sample ring (512 pairs)
ROWS = [1, 2, 3, 15, 16, 17, 31, 32, 33, 61, 62, 63, 64, 65, 255, 256, 257, 287, 319, 1023, 1024,
        1025, 1057, 1087]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("cols", [1, 7, 8, 255, 256, 257, 1023, 1024, 1025, 1281, 2049])
@pytest.mark.parametrize("mode", MODES)
def test_block_edges(env, mode, cols, dtype):
    rng = np.random.default_rng([cols, mode[0], mode[1]])
    centroid = _signal(rng, cols, dtype)
    members = [_signal(rng, L, dtype) for L in ROWS]
    torch, api = env
    ds = api.DeviceSeries.from_host(members)
    c = torch.from_numpy(centroid).cuda()
    mean, counts, delta, _ = api.dba_round(c, ds, *mode)
    w_mean, w_counts, _, w_delta = O.dba_update(centroid, members, *mode, fma_mode=1)
    assert mean.cpu().numpy().tobytes() == w_mean.tobytes()
    assert np.array_equal(counts.cpu().numpy().astype(np.uint32), w_counts)
    assert delta == w_delta or (np.isnan(delta) and np.isnan(w_delta))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("mode", MODES[::2])
def test_more_swaths_than_blocks(env, mode, dtype):
    rng = np.random.default_rng(77)
    centroid = _signal(rng, 2060, dtype)   # three swaths, the last 12 columns wide
    kinds = [_signal(rng, L, dtype) for L in range(600, 1000, 17)]
    members = kinds * 18                   # 432 members, 1296 swaths
    want = O.member_ranges(centroid, kinds, *mode, fma_mode=1)
    for _ in range(3):
        got = _ranges(env, centroid, members, *mode)
        for k in range(len(members)):
            assert np.array_equal(got[k], want[k % len(kinds)]), f"member {k}"


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_mixed_swath_counts(env, dtype):
    # open end, centroid shorter: the members take the columns, one to four
    # swaths each, and only the last swaths share a turn
    rng = np.random.default_rng(5)
    centroid = _signal(rng, 300, dtype)
    kinds = [_signal(rng, L, dtype) for L in (100, 299, 301, 1000, 1024, 1025, 2048, 2049, 3073, 4000)]
    members = kinds * 60
    want = O.member_ranges(centroid, kinds, 0, 1, fma_mode=1)
    got = _ranges(env, centroid, members, 0, 1)
    for k in range(len(members)):
        assert np.array_equal(got[k], want[k % len(kinds)]), f"member {k}"
