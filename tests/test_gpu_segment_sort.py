"""Segment medians from the exchange sort's own kernel: blocks with negative
zeros, and blocks too long for the rank sort's copy, beside blocks that have
neither, against the CPU oracle bit for bit; up to the longest minimum segment
length that a block's shared memory takes."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

LONGEST = {np.float32: 534, np.float64: 267}


@pytest.fixture(scope="module")
def api():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opendba_b200 import api as A
    from opendba_b200 import build
    build.build_library()
    return A


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("minseg", [1, 4, 9, 128, 130, 131, 190, -1, 0])
def test_mixed_blocks(api, minseg, dtype):
    minseg = LONGEST[dtype] + minseg if minseg <= 0 else minseg
    rng = np.random.default_rng(minseg)
    spb = 256 * ((minseg + 2) // 3)
    n = min(6 * spb + 37, 16000)
    x = (np.repeat(rng.normal(0, 1, n // 9 + 1), 9)[:n] + rng.normal(0, 0.1, n)).astype(dtype)
    zeros = x.copy()
    zeros[rng.random(n) < 0.4] = dtype(0.0)
    zeros[rng.random(n) < 0.2] = dtype(-0.0)
    part = x.copy()
    part[: min(n, spb) // 2 : 3] = dtype(-0.0)   # the first block only
    series = [x, zeros, part, x[: n // 3], zeros[:5]]
    got = api.segment_host(series, minseg)
    want = O.segment(series, minseg)
    for s, g, w in zip(series, got, want):
        assert len(g) == len(w), len(s)
        assert g.tobytes() == np.ascontiguousarray(w, dtype=dtype).tobytes(), len(s)
