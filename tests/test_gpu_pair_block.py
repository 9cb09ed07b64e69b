"""The block-per-swath pair plan over task lists, against the CPU oracle bit for
bit: either series the longer one (without an open end the shorter one takes
the rows), second series longer than the longest first one (the launch sizes
its swaths by the first ones), rows and columns at the edges of lanes, warps
and swaths, the open-end shortcut included."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

PIPELINE = 3
TASK = np.dtype([("first", "<u4"), ("second", "<u4"), ("out", "<u8")])
LENS = [1, 2, 3, 17, 40, 255, 256, 257, 700, 1023, 1024, 1025, 1300, 2048, 2049, 3100]


@pytest.fixture(scope="module")
def env():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opendba_b200 import _native, api, build
    build.build_library()
    return torch, api, _native


def _run(env, series, pairs, os_, oe, max_len):
    torch, api, native = env
    ds = api.DeviceSeries.from_host(series)
    sfx = {4: "f32", 8: "f64"}[ds.dtype.itemsize]
    tasks = np.empty(len(pairs), dtype=TASK)
    tasks["first"] = [p[0] for p in pairs]
    tasks["second"] = [p[1] for p in pairs]
    tasks["out"] = (np.arange(len(pairs), dtype=np.uint64) | np.uint64(os_ << 62) | np.uint64(oe << 63))
    d_tasks = torch.from_numpy(tasks.view(np.uint8)).cuda()
    out = torch.full((len(pairs),), float("nan"), dtype=ds.data.dtype, device="cuda")
    ws = torch.empty(native.lib().odba_dtw_pairwise_workspace_bytes(ds.dtype.itemsize, max_len),
                     dtype=torch.uint8, device="cuda")
    key = (ds.dtype.itemsize, max_len.bit_length() - 1, len(pairs).bit_length() - 1)
    assert native.lib().odba_tune_set(*key, PIPELINE) == 0
    try:
        native.call(f"odba_dtw_pairlist_{sfx}", ds.data.data_ptr(), ds.offsets.data_ptr(),
                    ds.lens.data_ptr(), d_tasks.data_ptr(), len(pairs), max_len, out.data_ptr(),
                    ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    finally:
        native.lib().odba_tune_set(*key, 0)
    err = ws[8:12].cpu().numpy().view(np.uint32)[0]
    assert err == 0
    return out.cpu().numpy()


def _check(env, series, pairs, mode, max_len):
    got = _run(env, series, pairs, *mode, max_len)
    for i, (a, b) in enumerate(pairs):
        want = O.dtw_pair(series[a], series[b], *mode, fma_mode=1)
        want = np.asarray(want, dtype=got.dtype)
        assert got[i].tobytes() == want.tobytes(), (len(series[a]), len(series[b]), got[i], want)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("mode", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_every_order_of_lengths(env, mode, dtype):
    rng = np.random.default_rng(31)
    series = [np.cumsum(rng.standard_normal(L)).astype(dtype) for L in LENS]
    # single-row matrices with a free end read a word the reference leaves
    # unset: their rows start at 2
    pairs = [(a, b) for a in range(len(LENS)) for b in range(len(LENS))
             if a != b and (LENS[a] > 1 or mode == (0, 0))]
    _check(env, series, pairs, mode, max(LENS))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("mode", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_second_series_longer_than_max_len(env, mode, dtype):
    rng = np.random.default_rng(8)
    short = [2, 31, 500, 1000]
    long = [1025, 2048, 2100, 4200, 5000]
    series = [np.cumsum(rng.standard_normal(L)).astype(dtype) for L in short + long]
    # copies of a first series' end: the shortcut's last-row minimum
    series.append(np.concatenate([series[2], np.full(2500, series[2][-1], dtype=dtype)]).astype(dtype))
    pairs = [(a, len(short) + b) for a in range(len(short)) for b in range(len(long) + 1)]
    _check(env, series, pairs, mode, max(short))
