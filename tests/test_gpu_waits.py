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
    assert _native.lib().odba_selftest_wait_timeout(1_000_000, None) == 6  # loads the kernels
    return _native.lib()


def _seconds(lib, limit_s):
    """The quickest of three calls (a call now and then is half a second late)."""
    best = 1e9
    for _ in range(3):
        t0 = time.perf_counter()
        rc = lib.odba_selftest_wait_timeout(int(limit_s * 1e9), None)
        best = min(best, time.perf_counter() - t0)
        assert rc == 6, lib.odba_last_error()
    return best


@pytest.mark.parametrize("limit_s", [0.02, 0.3])
def test_pipeline_wait_runs_out_at_its_limit(lib, limit_s):
    dt = _seconds(lib, limit_s)
    assert limit_s < dt
    # the waits of a sweep that has given up do not add up
    assert dt < 6 * limit_s + 0.5


def test_wait_inside_a_block_runs_out_and_reports(lib):
    # the compute warps' own wait, without a neighbouring block: four limits after
    # the pipeline's one
    assert _seconds(lib, 0.2) > 0.9
