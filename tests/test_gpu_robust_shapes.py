"""The robust statistics over arrays of few columns, few rows and tiny slices,
whose tiles are narrower, wider or not used, against the oracle, bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

from tests.conftest import bits

pytestmark = pytest.mark.gpu

SHAPES = [((700, 1), (5, 1)), ((700, 2), (5, 2)), ((401, 3), (9, 2)), ((300, 5), (4, 3)), ((90, 17), (7, 7)),
          ((60, 40, 3), (5, 5, 1)), ((200, 2, 2), (3, 2, 2)), ((150, 1, 3), (5, 1, 3)), ((90, 4, 5), (1, 3, 3)),
          ((2, 900), (2, 9)), ((3, 700), (3, 3)), ((7, 530), (5, 5)), ((1, 900), (3, 11)), ((33, 33), (11, 11)),
          ((2, 1, 600), (1, 1, 25)), ((5,), (3,)), ((1, 1), (3, 3)), ((3, 2, 1), (3, 3, 3))]


@pytest.mark.parametrize("kind, options", (("mad", dict(parameter=1.4826)), ("sigma_mode", dict(maxiters=None)),
                                           ("mode", dict(estimator="sex", pearson=2.5))))
def test_narrow_arrays_match_oracle(gpu, oracle, kind, options) -> None:
    from ndfiltrs_gb300 import _core

    for i, (shape, size) in enumerate(SHAPES):
        rng = np.random.default_rng(i)
        values = (1000 + 10 * rng.normal(size=shape)).astype(np.float32)
        values[rng.random(shape) < 0.03] = np.nan
        values[rng.random(shape) < 0.02] = 50000
        mode = ("reflect", "constant", "nearest", "mirror", "wrap")[i % 5]
        ignore_inf = kind != "mad"
        with _core.Plan(shape, np.float32, kind, size, mode=[mode] * len(shape), cval=990.0, omit_nan=True,
                        ignore_inf=ignore_inf, robust=options) as plan:
            actual = plan.run_host(values)
        expected = oracle.robust_filter(values, kind, size, mode=mode, cval=990.0, omit_nan=True,
                                        ignore_inf=ignore_inf, **options)
        np.testing.assert_array_equal(bits(actual), bits(expected), err_msg=str((shape, size)))
