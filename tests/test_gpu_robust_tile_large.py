"""The robust tile kernel over arrays large enough for tiles of 512 outputs (four
to a thread, which reuses its column of samples), against the oracle, bit for bit, in
strips of rows at the tiles' edges and the array's."""

from __future__ import annotations

import numpy as np
import pytest

from tests.conftest import bits

pytestmark = pytest.mark.gpu


# 600 x 717: 874 tiles of 32 x 16, more than the 608 that 152 SMs take before tiles
# are cut to 128 outputs.
@pytest.mark.parametrize("size", ((3, 3), (5, 5), (6, 4), (7, 7), (9, 9), (8, 16)))
@pytest.mark.parametrize("kind, options", (
    ("mad", dict(parameter=1.4826)), ("mode", dict(estimator="sex", pearson=2.5)),
    ("sigma_mode", dict(maxiters=None)), ("sigma_mean", dict(center="mean", spread="mad", maxiters=5))))
def test_large_tiles_match_oracle(gpu, oracle, kind, options, size) -> None:
    from ndfiltrs_gb300 import _core

    shape = (600, 717)
    rng = np.random.default_rng(size[0] * 100 + size[1])
    values = 1000 + 10 * rng.normal(size=shape)
    values = np.where(rng.random(shape) < 0.01, rng.uniform(2000, 60000, shape), values)
    values[rng.random(shape) < 0.03] = np.nan
    values[rng.random(shape) < 0.01] = np.inf
    values[300:320, 200:260] = np.nan
    values = values.astype(np.float32)
    clip = kind.startswith("sigma")
    with _core.Plan(shape, np.float32, kind, size, mode=["mirror"] * 2, omit_nan=True, ignore_inf=clip,
                    robust=options) as plan:
        actual = plan.run_host(values)
    for a, b in ((0, 20), (24, 40), (296, 324), (584, 600)):
        low, high = max(0, a - size[0]), min(shape[0], b + size[0])
        expected = oracle.robust_filter(values[low:high], kind, size, mode="mirror", omit_nan=True, ignore_inf=clip,
                                        **options)[a - low:b - low]
        np.testing.assert_array_equal(bits(actual[a:b]), bits(expected), err_msg=str((a, b)))
