"""A first series longer than the max_len a launch was sized for: its pairs are
NaN under every plan, the other pairs are what they are without it, and nothing
is written past the workspace."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

TASK = np.dtype([("first", "<u4"), ("second", "<u4"), ("out", "<u8")])
GUARD = 1 << 20


@pytest.fixture(scope="module")
def env():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opendba_b200 import _native, api, build
    build.build_library()
    return torch, api, _native


@pytest.mark.parametrize("pairlist", [False, True])
@pytest.mark.parametrize("plan", [0, 1, 2, 3])
@pytest.mark.parametrize("mode", [(0, 0), (0, 1), (1, 0)])
@pytest.mark.parametrize("max_len,long", [(300, 1500), (1200, 5000)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_too_long_first_series(env, dtype, max_len, long, mode, plan, pairlist):
    torch, api, native = env
    lib = native.lib()
    rng = np.random.default_rng(5)
    lens = [200, long, max_len, 257, long + 77, 150]
    series = [np.cumsum(rng.standard_normal(L)).astype(dtype) for L in lens]
    ds = api.DeviceSeries.from_host(series)
    elem, sfx = ds.dtype.itemsize, {4: "f32", 8: "f64"}[ds.dtype.itemsize]
    pairs = [(i, j) for i in range(len(lens)) for j in range(i + 1, len(lens))]
    nbytes = lib.odba_dtw_pairwise_workspace_bytes(elem, max_len)
    ws = torch.full((nbytes + GUARD,), 0x5A, dtype=torch.uint8, device="cuda")
    out = torch.zeros(len(pairs), dtype=ds.data.dtype, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    key = (elem, max_len.bit_length() - 1, len(pairs).bit_length() - 1)
    assert lib.odba_tune_set(*key, plan) == 0
    try:
        if pairlist:
            tasks = np.empty(len(pairs), dtype=TASK)
            tasks["first"], tasks["second"] = zip(*pairs)
            tasks["out"] = (np.arange(len(pairs), dtype=np.uint64) | np.uint64(mode[0] << 62)
                            | np.uint64(mode[1] << 63))
            d_tasks = torch.from_numpy(tasks.view(np.uint8)).cuda()
            native.call(f"odba_dtw_pairlist_{sfx}", ds.data.data_ptr(), ds.offsets.data_ptr(),
                        ds.lens.data_ptr(), d_tasks.data_ptr(), len(pairs), max_len,
                        out.data_ptr(), ws.data_ptr(), nbytes, stream)
        else:
            native.call(f"odba_dtw_pairwise_{sfx}", ds.data.data_ptr(), ds.offsets.data_ptr(),
                        ds.lens.data_ptr(), len(lens), max_len, *mode, out.data_ptr(),
                        ws.data_ptr(), nbytes, stream)
    finally:
        lib.odba_tune_set(*key, 0)
    got = out.cpu().numpy()
    assert bool((ws[nbytes:] == 0x5A).all())
    for k, (i, j) in enumerate(pairs):
        if lens[i] > max_len:
            assert np.isnan(got[k]), (i, j)
        else:
            want = np.asarray(O.dtw_pair(series[i], series[j], *mode, fma_mode=1), dtype=dtype)
            assert got[k].tobytes() == want.tobytes(), (i, j)
