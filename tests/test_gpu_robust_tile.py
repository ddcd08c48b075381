"""The robust tile kernel (float32 windows of up to 128 samples) against the
oracle, bit for bit: every network width and the sizes next to it, tile edges
and ragged arrays of rank 1 to 3, and samples that exercise each of its
decisions: ties and quantized values (equal deviations), values around zero
(wide spans of set bits), spreads of one unit in the last place, mixed
magnitudes, infinities and windows with few samples."""

from __future__ import annotations

import numpy as np
import pytest

from tests.conftest import bits

pytestmark = pytest.mark.gpu


def _samples(style, shape, seed):
    rng = np.random.default_rng(seed)
    noise = rng.normal(size=shape)
    if style == "frame":
        x = 1000 + 10 * noise
        x = np.where(rng.random(shape) < 0.02, rng.uniform(2000, 60000, shape), x)
        x[rng.random(shape) < 0.03] = np.nan
        x[rng.random(shape) < 0.01] = np.inf
    elif style == "integers":
        x = np.round(3 * noise)
        x[rng.random(shape) < 0.05] = 40
    elif style == "zero":
        x = noise * np.exp(2 * rng.normal(size=shape))
        x[rng.random(shape) < 0.1] = -0.0
    elif style == "ulps":
        x = (1 + rng.integers(0, 3, shape) * 2.0 ** -23) * 1000
    else:  # "mixed"
        x = noise * 10.0 ** rng.integers(-30, 30, shape)
        x[rng.random(shape) < 0.2] = -np.inf
    return x.astype(np.float32)


CASES = [
    ("mad", dict(parameter=1.4826)),
    ("mad", dict(parameter=1.0)),
    ("mode", dict(estimator="sex", pearson=2.5)),
    ("mode", dict(estimator="iraf", pearson=3.0)),
    ("sigma_mode", dict(sigma_lower=3.0, sigma_upper=3.0, maxiters=None)),
    ("sigma_mean", dict(sigma_lower=0.5, sigma_upper=1.0, maxiters=3, center="mean")),
    ("sigma_mean", dict(sigma_lower=2.0, sigma_upper=2.5, maxiters=5, center="mean", spread="mad")),
    ("sigma_median", dict(sigma_lower=1.5, sigma_upper=1.5, maxiters=None, spread="mad")),
]
# (shape, size): volumes 1, 2 and around each network width; 512- and
# 128-output tiles, partial ones, single rows, lines and cubes.
WINDOWS = [((37, 41), (1, 1)), ((16, 33), (1, 2)), ((37, 41), (3, 3)), ((5, 70), (2, 5)), ((1, 600), (1, 16)),
           ((600,), (17,)), ((17, 64), (5, 5)), ((33, 31), (2, 13)), ((40, 32), (4, 8)), ((9, 45), (3, 11)),
           ((35, 37), (7, 7)), ((20, 35), (5, 10)), ((33, 33), (8, 8)), ((130,), (65,)), ((34, 40), (9, 9)),
           ((3, 19, 33), (2, 5, 8)), ((5, 9, 40), (3, 3, 3)), ((19, 40), (16, 8)), ((18, 36), (43, 3))]


@pytest.mark.parametrize("style", ("frame", "integers", "zero", "ulps", "mixed"))
def test_tile_kernel_matches_oracle(gpu, oracle, style) -> None:
    from ndfiltrs_gb300 import _core

    for i, (shape, size) in enumerate(WINDOWS):
        values = _samples(style, shape, seed=i)
        mode = ("reflect", "constant", "nearest", "mirror", "wrap")[i % 5]
        for kind, options in CASES:
            clip = kind.startswith("sigma")
            for omit in (True,) if clip else (True, False):
                with _core.Plan(shape, np.float32, kind, size, mode=[mode] * len(shape), cval=2.5, omit_nan=omit,
                                ignore_inf=clip, robust=options) as plan:
                    actual = plan.run_host(values)
                expected = oracle.robust_filter(values, kind, size, mode=mode, cval=2.5, omit_nan=omit,
                                                ignore_inf=clip, **options)
                np.testing.assert_array_equal(bits(actual), bits(expected), err_msg=str((shape, size, kind, options)))
