"""Sigma clipping of data of few values (windows whose MAD is zero, and whose mean lies
among the samples or between them) in the tile kernel against the oracle, bit for
bit."""

from __future__ import annotations

import numpy as np
import pytest

from tests.conftest import bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", ((3, 3), (4, 4), (5, 7), (9, 9)))
@pytest.mark.parametrize("kind", ("sigma_mean", "sigma_median", "sigma_mode"))
@pytest.mark.parametrize("center", ("mean", "median"))
def test_few_values_match_oracle(gpu, oracle, kind, center, size) -> None:
    from ndfiltrs_gb300 import _core

    shape = (70, 90)
    rng = np.random.default_rng(size[1])
    for style in range(4):
        if style == 0:  # mostly zeros
            values = (rng.random(shape) < 0.15) * 1.0
        elif style == 1:  # symmetric about the mode: the mean is a sample
            values = 7.5 + np.where(rng.random(shape) < 0.2, rng.choice((-3.0, 3.0), shape), 0.0)
        elif style == 2:
            values = np.where(rng.random(shape) < 0.6, -0.0, rng.integers(-2, 3, shape)) * 1e-3
        else:
            values = np.where(rng.random(shape) < 0.7, 1000.0, 1000.0 + 10.0 ** rng.integers(-3, 20, shape))
        values = values.astype(np.float32)
        values[rng.random(shape) < 0.05] = np.nan
        for maxiters in (None, 1):
            options = dict(sigma_lower=2.0, sigma_upper=3.0, center=center, spread="mad", maxiters=maxiters)
            with _core.Plan(shape, np.float32, kind, size, omit_nan=True, ignore_inf=True, robust=options) as plan:
                actual = plan.run_host(values)
            expected = oracle.robust_filter(values, kind, size, omit_nan=True, ignore_inf=True, **options)
            np.testing.assert_array_equal(bits(actual), bits(expected), err_msg=str((style, maxiters)))
