"""Stripe mode takes the workspace it is given: members and stripes go side by
side where there is room, one after the other where there is not, with the same
results; the size of one member at a time (its edges, its checkpoint rows and the
moves of one stripe) is enough."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = 64


@pytest.fixture(scope="module")
def env():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opendba_b200 import _native, api, build
    build.build_library()
    return torch, api, _native


def _one_member(elem, lens, lc, oe):
    """Bytes of one member at a time: see the parts named above, a 256-byte
    header, a progress word per swath, and 2.5 MB for the reducer's tables (two
    64-sample edges per resident warp) of this few members."""
    flip = [oe and lc < n for n in lens]
    rows = max(lc if f else n for f, n in zip(flip, lens))
    cols = max(n if f else lc for f, n in zip(flip, lens))
    width = 1024 if elem == 4 else 512
    swaths = -(-cols // width)
    edges = max(swaths - 1, 1) * ((rows + 95) // 32 * 32) * elem
    ckpt = (rows // ROWS + 1) * swaths * width * elem
    moves = ((rows + 1) // 2 + 32) * 512 * (2 if oe and elem == 8 else 1)
    ranges = len(lens) * lc * 8
    extra = len(lens) * lc * 4 if oe else 0
    return edges + ckpt + moves + ranges + extra + 256 + swaths * 24 + int(2.5 * 2 ** 20)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("mode", [(0, 0), (0, 1), (1, 1)])
def test_any_workspace_gives_the_same_round(env, mode, dtype):
    torch, api, native = env
    rng = np.random.default_rng(17)
    lens = [6000, 5100, 7400, 4096, 900]
    series = [np.cumsum(rng.standard_normal(L)).astype(dtype) for L in lens]
    ds = api.DeviceSeries.from_host(series)
    cen = torch.from_numpy(series[1].copy()).cuda()
    elem, lc = ds.dtype.itemsize, len(series[1])
    h = np.array(lens, dtype=np.uint64)
    full = native.lib().odba_dba_round_stripe_workspace_bytes(
        elem, h.ctypes.data_as(ctypes.c_void_p), len(lens), lc, *mode, ROWS)
    want = api.dba_round(cen, ds, *mode)

    def same(a, b):  # bit for bit: an index that receives nothing is NaN
        return a[0].cpu().numpy().tobytes() == b[0].cpu().numpy().tobytes() and torch.equal(a[1], b[1])

    def run(nbytes):
        ws = torch.full((nbytes + 4096,), 0x5A, dtype=torch.uint8, device="cuda")
        got = api.dba_round(cen, ds, *mode, workspace=ws[:nbytes], stripe_rows=ROWS)
        assert bool((ws[nbytes:] == 0x5A).all())
        return got

    first = run(full)
    if not mode[1]:  # (with an open end a stripe's height has rules of its own)
        assert same(first, want)
    small = _one_member(elem, lens, lc, mode[1])
    assert small < full // 2
    taken = 0
    for nbytes in [full * k // 16 for k in range(15, 0, -1)] + [small]:
        if nbytes < small:
            continue
        got = run(nbytes)
        assert same(got, first) and got[2] == first[2]
        taken += 1
    assert taken >= 5
    with pytest.raises(native.OdbaError):
        run(small // 4)


def _least(run, high, native):
    """The smallest workspace a round takes (nothing smaller is launched)."""
    low = 0
    while high - low > 4096:
        mid = (low + high) // 2
        try:
            run(mid)
            high = mid
        except native.OdbaError:
            low = mid
    return high


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e30])
def test_walks_that_fail_leave_the_same_samples(env, value, dtype):
    # with the least workspace a member's path is walked cell by cell, with more
    # row by row; NaN and infinite costs lead some walks off the first column
    torch, api, native = env
    rng = np.random.default_rng(23)
    lens = [2200, 700, 1500, 3, 40, 1100, 2500, 65]
    series = [np.cumsum(rng.standard_normal(L)).astype(dtype) for L in lens]
    for s in series:
        if rng.random() < 0.6:
            s[rng.integers(0, len(s), size=2)] = value
    ds = api.DeviceSeries.from_host(series)
    for c in (2, 5, 6):
        for open_both in (0, 1):
            cen = torch.from_numpy(series[c].copy()).cuda()

            def run(nbytes):
                ws = None if nbytes is None else torch.empty(nbytes, dtype=torch.uint8, device="cuda")
                got = api.dba_round(cen, ds, open_both, 0, workspace=ws, stripe_rows=ROWS)
                return got[0].cpu().numpy().tobytes(), got[1].cpu().numpy().tobytes(), got[2]

            assert run(None) == run(_least(run, 64 << 20, native)), (c, open_both)
