"""The bounded waits of the block sweep, made to run out with short limits on a
word that nothing raises: the kernel returns by itself and says so."""
import time

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opendba_b200 import _native, build
    build.build_library()
    assert _native.lib().odba_selftest_wait_timeout(1_000_000, None) == 6  # loads the kernel
    return _native.lib()


@pytest.mark.parametrize("limit_s", [0.02, 0.3])
def test_pipeline_wait_runs_out_at_its_limit(lib, limit_s):
    t0 = time.perf_counter()
    rc = lib.odba_selftest_wait_timeout(int(limit_s * 1e9), None)
    dt = time.perf_counter() - t0
    assert rc == 6, lib.odba_last_error()
    assert limit_s < dt
    # the waits of a sweep that has given up do not add up
    assert dt < 6 * limit_s + 0.5
