"""The segmentation kernel's two DP forms and its rank sort, at the sizes where
they change over, against the CPU oracle bit for bit."""
import numpy as np
import pytest

from opendba_b200 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _signals(minseg, kind, dtype):
    rng = np.random.default_rng([minseg, len(kind)])
    dw = (minseg + 2) // 3
    spb = 256 * dw
    # a block and its edges, a few samples, and partial blocks whose longest
    # segment lies around the fast form's limits (148 and 196 points)
    lens = [1, 2, 2 * dw + 1, spb - 1, spb, spb + 1, 147 * dw, 148 * dw + 1, 149 * dw,
            195 * dw, 196 * dw, 197 * dw + dw // 2, 2 * spb + 32 * dw]
    out = []
    for L in lens:
        if kind == "steps":
            x = np.repeat(rng.normal(90, 12, L // 7 + 1), 7)[:L] + rng.normal(0, 2, L)
        elif kind == "high":   # sums past the fast form's range: almost every point at the top
            x = np.full(L, 1000.0) + rng.normal(0, 0.01, L)
            x[: max(1, L // 300)] = 0.0
        elif kind == "flat":
            x = np.zeros(L)
        else:                  # ties and both zeros: the exchange sort, not ranks
            x = rng.integers(-1, 2, L).astype(np.float64)
            x[rng.random(L) < 0.3] = -0.0
        # the block range is taken over whole groups of 32 points; a later point
        # outside it overflows the 8-bit conversion, which the oracle restates as
        # a clamp and the device does not: keep those points inside the range
        points = (L % spb) // dw
        if points % 32 and points >= 32:
            x[L - L % spb + points // 32 * 32 * dw:] = x[L - L % spb]
        out.append(x.astype(dtype))
    return out


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("minseg", [2, 3, 4, 5, 9, 40])
@pytest.mark.parametrize("kind", ["steps", "high", "flat", "zeros"])
def test_segment_forms_match_oracle(minseg, kind, dtype):
    series = _signals(minseg, kind, dtype)
    got = api.segment_host(series, minseg)
    want = O.segment(series, minseg)
    for g, w in zip(got, want):
        assert len(g) == len(w)
        assert g.tobytes() == np.ascontiguousarray(w, dtype=dtype).tobytes()
