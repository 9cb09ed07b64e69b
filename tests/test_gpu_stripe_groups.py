"""The stripe-mode round with more members than run side by side and more
stripes than one group holds, against the full-path round (without an open end
the two are equal bit for bit) and, with an open end, against one member at a
time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opendba_b200 import api, build
    build.build_library()
    return torch, api


def _signal(rng, L, dtype):
    return (np.repeat(rng.normal(0, 1, L // 9 + 1), 9)[:L] + rng.normal(0, 0.1, L)).astype(dtype)


def _host(r):
    return r[0].cpu().numpy().tobytes(), r[1].cpu().numpy().tobytes(), r[2]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("os_", [0, 1])
@pytest.mark.parametrize("cols,lens,rows", [
    (9300, [1, 2, 33, 300, 511, 512, 513, 1025, 1700, 2600, 2601], 512),  # 11 members, 2 groups
    (17000, [12000, 15555, 9001], 1024),                                  # 3 groups, walks across them
    (1024, [5000, 16385], 4096),
])
def test_stripe_groups_equal_full_path(env, cols, lens, rows, os_, dtype):
    torch, api = env
    rng = np.random.default_rng([cols, os_])
    cen = torch.from_numpy(_signal(rng, cols, dtype)).cuda()
    ds = api.DeviceSeries.from_host([_signal(rng, L, dtype) for L in lens])
    full = api.dba_round(cen, ds, os_, 0, with_paths=True)
    plain = api.dba_round(cen, ds, os_, 0, stripe_rows=rows)
    listed = api.dba_round(cen, ds, os_, 0, with_paths=True, stripe_rows=rows)
    assert _host(plain) == _host(full) and _host(listed) == _host(full)
    for a, b in zip(listed[3], full[3]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("os_", [0, 1])
def test_stripe_open_end_side_by_side(env, os_, dtype):
    # members of both orientations in one batch: every path is the one the
    # member has when it is the only member
    torch, api = env
    rng = np.random.default_rng(5)
    cen = torch.from_numpy(_signal(rng, 3300, dtype)).cuda()
    members = [_signal(rng, L, dtype) for L in [40, 900, 1500, 2500, 3299, 3300, 3301, 4200, 5000, 700]]
    ds = api.DeviceSeries.from_host(members)
    got = api.dba_round(cen, ds, os_, 1, with_paths=True, stripe_rows=256)[3]
    for k, m in enumerate(members):
        one = api.dba_round(cen, api.DeviceSeries.from_host([m]), os_, 1, with_paths=True,
                            stripe_rows=256)[3][0]
        assert np.array_equal(got[k], one), f"member {k}"
