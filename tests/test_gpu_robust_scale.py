"""The MAD's scale against the oracle, bit for bit: scales down to the smallest,
with deviations that are exact in float32 and large enough for the product to be
a normal float."""

from __future__ import annotations

import numpy as np
import pytest

from tests.conftest import bits

pytestmark = pytest.mark.gpu

SCALES = (1.4826, 1.4826e-28, 1.4826e-30, 2.0 ** -100, 2.0 ** -100 * (1 + 2.0 ** -30), 7.8886e-31, 1.4826e-36, 3.3e-38,
          1e-40, 1e-300, 5e-324, 0.0, -0.0, 1e37, 1e300)


@pytest.mark.parametrize("size", ((3, 3), (4, 4), (9, 9)))
def test_mad_scales_match_oracle(gpu, oracle, size) -> None:
    from ndfiltrs_gb300 import _core

    rng = np.random.default_rng(size[0])
    values = (2.0 ** 40 + rng.integers(-2 ** 20, 2 ** 20, (90, 150)) * 2.0 ** 20).astype(np.float32)
    values[:8, :20] = 2.0 ** 40  # deviations of zero
    for scale in SCALES:
        with _core.Plan(values.shape, np.float32, "mad", size, omit_nan=True, robust=dict(parameter=scale)) as plan:
            actual = plan.run_host(values)
        expected = oracle.robust_filter(values, "mad", size, omit_nan=True, parameter=scale)
        np.testing.assert_array_equal(bits(actual), bits(expected), err_msg=str(scale))
