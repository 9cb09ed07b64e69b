"""Large rounds, whose path DTW is swept by one warp per swath, against the CPU
oracle bit for bit: rows around its chunks of 32 pairs, columns around its lane
widths (8, 16 and 32 columns per lane in a last swath) and swaths (1024 columns in
float, 512 in double), the path listing and the prefix chop's walk included."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

MODES = [(0, 0), (1, 0), (0, 1), (1, 1)]
ROWS = [1, 2, 3, 31, 32, 33, 62, 63, 64, 65, 66, 97, 127, 128, 129, 191, 257]


@pytest.fixture(scope="module")
def env():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opendba_b200 import _native, api, build
    build.build_library()
    return torch, api, _native


def _signal(rng, L, dtype):
    return (np.repeat(rng.normal(0, 1, L // 9 + 1), 9)[:L] + rng.normal(0, 0.1, L)).astype(dtype)


def _many(kinds, lc, dtype, open_end=0, leader=False):
    """Copies of the kinds in turn: more work, in swaths of the most rows, than the
    resident warps (1776 float, 1184 double) times what the rule asks."""
    flip = [leader or (open_end and lc < len(k)) for k in kinds]
    rows = np.array([lc if f else len(k) for f, k in zip(flip, kinds)])
    swaths = np.array([-(-(len(k) if f else lc) // 1024) for f, k in zip(flip, kinds)])
    wide = swaths.max() > 4
    need = (1776 * (1.5 if wide else 0.95)) if dtype == np.float32 else 1184 * (1.0 if wide else 0.7)
    n = int(need * rows.max() / (rows * swaths).mean()) + len(kinds)
    return [kinds[k % len(kinds)] for k in range(n)]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("cols", [1, 9, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 1281, 1537, 2049])
@pytest.mark.parametrize("mode", MODES)
def test_lane_and_chunk_edges(env, mode, cols, dtype):
    torch, api, _ = env
    rng = np.random.default_rng([cols, mode[0], mode[1]])
    centroid = _signal(rng, cols, dtype)
    kinds = [_signal(rng, L, dtype) for L in ROWS]
    members = _many(kinds, cols, dtype, mode[1])
    ds = api.DeviceSeries.from_host(members)
    got = api.dba_round_ranges(torch.from_numpy(centroid).cuda(), ds, *mode).cpu().numpy()
    want = O.member_ranges(centroid, kinds, *mode, fma_mode=1)
    for k in range(len(members)):
        assert np.array_equal(got[k], want[k % len(kinds)]), f"member {k}"


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("mode", MODES)
def test_whole_round_and_paths(env, mode, dtype):
    # open end: the longer members take the columns, one to four swaths each, and
    # the shortcut is checked on their edges
    torch, api, _ = env
    rng = np.random.default_rng([9, mode[0], mode[1]])
    centroid = _signal(rng, 300, dtype)
    lens = (40, 299, 301, 600, 1100, 1700, 2300, 3300) if mode[1] else (40, 250, 299, 300, 301, 410)
    kinds = [_signal(rng, L, dtype) for L in lens]
    if mode[1]:
        kinds.append(np.concatenate([centroid, np.full(2500, centroid[-1], dtype=dtype)]))
    members = _many(kinds, 300, dtype, mode[1])
    ds = api.DeviceSeries.from_host(members)
    c = torch.from_numpy(centroid).cuda()
    mean, counts, delta, _ = api.dba_round(c, ds, *mode)
    w_mean, w_counts, _, w_delta = O.dba_update(centroid, members, *mode, fma_mode=1)
    assert mean.cpu().numpy().tobytes() == w_mean.tobytes()
    assert np.array_equal(counts.cpu().numpy().astype(np.uint32), w_counts)
    assert delta == w_delta or (np.isnan(delta) and np.isnan(w_delta))
    listed = api.dba_round(c, ds, *mode, with_paths=True)
    assert listed[0].cpu().numpy().tobytes() == w_mean.tobytes()
    # the same members few at a time: a block per swath
    few = api.DeviceSeries.from_host(kinds)
    paths = api.dba_round(c, few, *mode, with_paths=True)[3]
    for k in range(len(members)):
        assert np.array_equal(listed[3][k], paths[k % len(kinds)]), f"member {k}"


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_prefix_chop_of_many_series(env, dtype):
    torch, api, native = env
    lib, elem = native.lib(), np.dtype(dtype).itemsize
    rng = np.random.default_rng(31)
    leader = _signal(rng, 260, dtype)
    kinds = [np.concatenate([leader + rng.normal(0, 0.05, 260).astype(dtype), _signal(rng, L, dtype)])
             for L in (1, 60, 300, 800, 1300, 2100)]

    def chop(series):
        ds = api.DeviceSeries.from_host(series, dtype=dtype)
        h = np.ascontiguousarray(ds.host_lens, dtype=np.uint64)
        hp = h.ctypes.data_as(ctypes.c_void_p)
        lead = torch.from_numpy(leader).cuda()
        ws = torch.empty(lib.odba_prefix_chop_workspace_bytes(elem, hp, ds.n, len(leader)),
                         dtype=torch.uint8, device="cuda")
        pos = torch.empty(ds.n, dtype=torch.int64, device="cuda")
        hist = torch.empty((ds.n, len(leader)), dtype=torch.int32, device="cuda")
        native.call(f"odba_prefix_chop_{'f32' if elem == 4 else 'f64'}", lead.data_ptr(), len(leader),
                    ds.data.data_ptr(), ds.offsets.data_ptr(), ds.lens.data_ptr(), hp, ds.n,
                    pos.data_ptr(), hist.data_ptr(), ws.data_ptr(), ws.numel(),
                    torch.cuda.current_stream().cuda_stream)
        return pos.cpu().numpy(), hist.cpu().numpy()

    few = chop(kinds)
    many = chop(_many(kinds, 260, dtype, leader=True))
    for k in range(len(many[0])):
        assert many[0][k] == few[0][k % len(kinds)]
        assert np.array_equal(many[1][k], few[1][k % len(kinds)])
