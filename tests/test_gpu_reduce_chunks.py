"""The ordered reducer's distribution of members over lanes against the CPU
oracle bit for bit: member counts around a lane per member, the members per
lane and the chunk of 128, with short members (many samples from one member at
one centroid index) and long ones (samples past the first of a range)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("count", [1, 2, 31, 32, 33, 64, 65, 96, 97, 127, 128, 129, 160, 161, 257])
def test_member_counts(count, dtype):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opendba_b200 import api, build
    build.build_library()
    rng = np.random.default_rng(count)
    centroid = rng.standard_normal(37).astype(dtype)
    members = [rng.standard_normal(int(rng.integers(2, 150))).astype(dtype) for _ in range(count)]
    mode = (0, count % 2)
    mean, counts, delta, _ = api.dba_round(torch.from_numpy(centroid).cuda(),
                                           api.DeviceSeries.from_host(members), *mode)
    w_mean, w_counts, _, w_delta = O.dba_update(centroid, members, *mode, fma_mode=1)
    assert mean.cpu().numpy().tobytes() == w_mean.tobytes()
    assert np.array_equal(counts.cpu().numpy().astype(np.uint32), w_counts)
    assert delta == w_delta
