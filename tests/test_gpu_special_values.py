"""Pairs with NaN, infinite and overflowing samples: every plan gives what the
cell rule gives in plain arithmetic.  Minima are fmin's in float (a NaN loses)
and compare-and-selects in double, in the order up, diagonal, left; the open-end
shortcut stops a pair only where the edge's last-row value equals the minimum,
which a NaN never does."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PLANS = {"whole": 1, "half": 2, "pipeline": 3}


@pytest.fixture(scope="module")
def env():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opendba_b200 import _native, api, build
    build.build_library()
    return torch, api, _native


def _min2(dtype):
    if dtype == np.float32:
        return lambda a, b: b if a != a or b < a else a
    return lambda a, b: b if b < a else a


def distance(x, y, oe, dtype):
    """One pair without open start.  Small integers and special values: every
    product and sum of finite costs is exact, so no fused rounding matters."""
    big = float(np.finfo(dtype).max)
    min2 = _min2(dtype)
    top = float("inf") if dtype == np.float64 else big

    def cell(d, m):
        v = d * d + m
        # a float cost past the type's range is infinite
        return math.inf if dtype == np.float32 and v > top else v

    xs, ys = [float(v) for v in x], [float(v) for v in y]
    m, n = len(xs), len(ys)
    floor = 0 if dtype == np.float32 else 512
    left_col = [big] * m
    for c in range(n):
        col = []
        up = big
        diag_in = 0.0 if c == 0 else big
        for r in range(m):
            d = xs[r] - ys[c]
            diag = diag_in if r == 0 else left_col[r - 1]
            left = left_col[r]
            if oe and m >= 2 and r == m - 1:
                if c > 0 and c % 1024 == 0:
                    v = min2(min2(cell(d, up), diag), left)
                else:
                    v = min2(cell(d, min2(up, diag)), left)
            else:
                v = cell(d, min2(min2(up, diag), left))
            col.append(v)
            up = v
        left_col = col
        if oe and (c + 1) % 1024 == 0 and c + 1 < n and c + 1 > m:
            emin = big
            for r in range(m):
                if r % 1024 >= floor:
                    emin = min2(emin, col[r])
            if col[-1] == emin:
                corner = big if m == 1 else col[-1]
                break
    else:
        corner = left_col[-1]
    with np.errstate(all="ignore"):
        v = np.sqrt(np.float32(corner))
        return dtype(v / np.float32(m)) if oe else dtype(v)


def _series(rng, lens, dtype, value, spots):
    out = []
    for k, L in enumerate(lens):
        a = rng.integers(-3, 4, size=L).astype(dtype)
        for s in spots:
            if rng.random() < 0.5:
                a[s if 0 <= s < L else -1] = value
        out.append(a)
    return out


def _same(a, b):
    return (np.isnan(a) and np.isnan(b)) or a.tobytes() == b.tobytes()


def _check(env, plan, dtype, mode, value, lens, seed):
    torch, api, native = env
    lib = native.lib()
    rng = np.random.default_rng(seed)
    series = _series(rng, lens, dtype, value, [-1, 1023, 5])
    ds = api.DeviceSeries.from_host(series)
    pairs = [(i, j) for i in range(len(lens)) for j in range(i + 1, len(lens))]
    key = (ds.dtype.itemsize, int(ds.max_len).bit_length() - 1, len(pairs).bit_length() - 1)
    assert lib.odba_tune_set(*key, PLANS[plan]) == 0
    try:
        got = api.pairwise(ds, *mode).cpu().numpy()
    finally:
        lib.odba_tune_set(*key, 0)
    for k, (i, j) in enumerate(pairs):
        want = distance(series[i], series[j], mode[1], dtype)
        assert _same(got[k], want), (lens[i], lens[j], got[k], want)


@pytest.mark.parametrize("plan", list(PLANS))
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e30])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_open_end(env, dtype, value, plan):
    _check(env, plan, dtype, (0, 1), value, [1, 3, 40, 1025, 1100, 2100], 7)


@pytest.mark.parametrize("plan", list(PLANS))
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e30])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_global_either_series_the_longer_one(env, dtype, value, plan):
    # the pipeline puts the shorter series on the rows
    _check(env, plan, dtype, (0, 0), value, [2100, 1100, 600, 40, 3, 1, 700, 1030], 9)
