"""Segmentation of blocks with points outside the range the block is quantised
by (it is taken over whole groups of 32 points, and the minimum only for the
first point where there is one group or none): both forms of the DP against the
CPU oracle bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


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
@pytest.mark.parametrize("minseg", [2, 3, 4, 5, 9, 40])
@pytest.mark.parametrize("scale", [0.5, 3.0, 1e3, 1e9])
def test_points_outside_the_block_range(api, scale, minseg, dtype):
    rng = np.random.default_rng([minseg, int(scale)])
    dw = (minseg + 2) // 3
    series = []
    for points in [1, 5, 31, 32, 33, 47, 63, 64, 65, 100, 131, 160, 199, 255]:
        x = np.repeat(rng.normal(0, 1, points * dw // 7 + 1), 7)[: points * dw]
        x = x + rng.normal(0, 0.1, len(x))
        # the last, partial group of points leaves the range upwards and downwards
        tail = points // 32 * 32 * dw
        x[tail:] += scale * rng.choice([-1.0, 1.0], size=len(x) - tail)
        series.append(x.astype(dtype))
    got = api.segment_host(series, minseg)
    want = O.segment(series, minseg)
    for s, g, w in zip(series, got, want):
        assert len(g) == len(w), len(s)
        assert g.tobytes() == np.ascontiguousarray(w, dtype=dtype).tobytes(), len(s)
