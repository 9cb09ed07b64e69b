"""The one-warp-per-pair plans over task lists, against the CPU oracle bit for
bit: rows at the edges of the 32-pair chunks, last columns at the edges of
lanes and of the partial and full swaths, every mode, the open-end shortcut
included."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

WHOLE, HALF = 1, 2
TASK = np.dtype([("first", "<u4"), ("second", "<u4"), ("out", "<u8")])
ROWS = [1, 2, 3, 62, 63, 64, 65, 66, 127, 128, 129, 1000]
COLS = [1, 3, 4, 5, 127, 128, 129, 260, 383, 385, 511, 512, 513, 900, 1024, 1025, 1153, 2048, 2050]


@pytest.fixture(scope="module")
def env():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opendba_b200 import _native, api, build
    build.build_library()
    return torch, api, _native


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("mode", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("plan", [WHOLE, HALF])
def test_edges_of_chunks_lanes_and_swaths(env, plan, mode, dtype):
    torch, api, native = env
    rng = np.random.default_rng(17)
    series = [np.cumsum(rng.standard_normal(L)).astype(dtype) for L in ROWS + COLS]
    # a constant tail: the shortcut's last-row minimum
    series.append(np.concatenate([series[len(ROWS) - 1],
                                  np.full(1500, series[len(ROWS) - 1][-1])]).astype(dtype))
    # single-row matrices with a free end read a word the reference leaves
    # unset: their rows start at 2
    pairs = [(a, len(ROWS) + b) for a in range(len(ROWS)) for b in range(len(COLS) + 1)
             if ROWS[a] > 1 or mode == (0, 0)]
    ds = api.DeviceSeries.from_host(series)
    tasks = np.empty(len(pairs), dtype=TASK)
    tasks["first"] = [p[0] for p in pairs]
    tasks["second"] = [p[1] for p in pairs]
    tasks["out"] = (np.arange(len(pairs), dtype=np.uint64)
                    | np.uint64(mode[0] << 62) | np.uint64(mode[1] << 63))
    d_tasks = torch.from_numpy(tasks.view(np.uint8)).cuda()
    out = torch.full((len(pairs),), float("nan"), dtype=ds.data.dtype, device="cuda")
    size = np.dtype(dtype).itemsize
    lib = native.lib()
    max_len = max(ROWS)
    ws = torch.empty(lib.odba_dtw_pairwise_workspace_bytes(size, max_len), dtype=torch.uint8,
                     device="cuda")
    key = (size, max_len.bit_length() - 1, len(pairs).bit_length() - 1)
    assert lib.odba_tune_set(*key, plan) == 0
    try:
        native.call(f"odba_dtw_pairlist_f{8 * size}", ds.data.data_ptr(), ds.offsets.data_ptr(),
                    ds.lens.data_ptr(), d_tasks.data_ptr(), len(pairs), max_len, out.data_ptr(),
                    ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    finally:
        lib.odba_tune_set(*key, 0)
    got = out.cpu().numpy()
    for i, (a, b) in enumerate(pairs):
        want = np.asarray(O.dtw_pair(series[a], series[b], *mode, fma_mode=1), dtype=dtype)
        assert got[i].tobytes() == want.tobytes(), (len(series[a]), len(series[b]), got[i], want)
