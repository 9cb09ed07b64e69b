"""Device scratch that the host-buffer entry points keep between calls: a bounded
amount of it, given back on request."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.fixture(scope="module")
def env():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opendba_b200 import _native, api, build
    build.build_library()
    return torch, api, _native


def _pass(api, n, length):
    series = [np.full(length, k % 3, dtype=np.float32) for k in range(n)]
    return api.medoid_pass_host(series, norm=0)[0]


def test_kept_scratch_is_bounded_and_given_back(env):
    torch, api, native = env

    def free():
        return torch.cuda.mem_get_info()[0]

    assert _pass(api, 6, 500).shape == (15,)
    native.check(native.lib().odba_scratch_release())
    before = free()
    assert _pass(api, 1, 150_000_000).shape == (0,)  # 600 MB of scratch
    assert before - free() <= 256 * MB + 64 * MB
    first = _pass(api, 400, 2000)
    native.check(native.lib().odba_scratch_release())
    assert before - free() <= 4 * MB
    assert _pass(api, 400, 2000).tobytes() == first.tobytes()
