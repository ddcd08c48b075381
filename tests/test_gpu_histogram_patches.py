"""The histogram kernel's box windows (patches of outputs that share a
threshold rank) against the oracle, bit for bit: window and patch edges (row
counts of one word, exactly 32 columns, a word and a bit), single rows and
columns, tiles larger and smaller than the array, deep windows; samples that
stress the threshold (ramps along each axis, steps, ties, few retained samples,
none) and every kind of order statistic under both policies."""

from __future__ import annotations

import numpy as np
import pytest

from tests.conftest import bits

pytestmark = pytest.mark.gpu

MODES = ("reflect", "constant", "nearest", "mirror", "wrap")


def _samples(style, shape, seed):
    rng = np.random.default_rng(seed)
    x = np.indices(shape).astype(np.float64)
    if style == "noise":
        v = rng.normal(size=shape)
        v[rng.random(shape) < 0.01] = np.nan
        v[rng.random(shape) < 0.01] = np.inf
    elif style == "ramps":
        v = sum((axis + 1) * 7.0 * x[axis] ** 1.5 * (-1) ** axis for axis in range(len(shape)))
    elif style == "ties":
        v = rng.integers(0, 3, shape).astype(np.float64)
        v[rng.random(shape) < 0.2] = -0.0
    elif style == "steps":
        v = np.where(x[-1] % 23 < 11, -1e30, 1e30) + rng.normal(size=shape)
    elif style == "sparse":
        v = np.where(rng.random(shape) < 0.97, np.nan, rng.normal(size=shape))
        v.ravel()[::11] = np.inf
    else:  # "empty"
        v = np.full(shape, np.nan)
        v.ravel()[-1] = 3.0
    return v


KINDS = [("median", {}), ("rank", dict(parameter=3)), ("percentile", dict(percentile=84.0)),
         ("percentile", dict(percentile=0.0)), ("min", {}), ("max", {})]
WINDOWS = [((70, 90), (11, 11)), ((41, 77), (3, 32)), ((37, 133), (12, 33)), ((66, 40), (65, 65)), ((130, 35), (33, 1)),
           ((9, 300), (1, 64)), ((3, 500), (2, 25)), ((700,), (33,)), ((33, 129), (13, 26)), ((1, 40), (5, 57)),
           ((4, 30, 37), (3, 5, 9)), ((7, 12, 70), (9, 17, 25)), ((2, 3, 40), (2, 2, 33))]


@pytest.mark.parametrize("dtype", (np.float32, np.float64))
@pytest.mark.parametrize("style", ("noise", "ramps", "ties", "steps", "sparse", "empty"))
def test_patches_match_oracle(gpu, oracle, style, dtype) -> None:
    from ndfiltrs_gb300 import _core

    _core.pin_kernel("histogram")
    try:
        for i, (shape, size) in enumerate(WINDOWS):
            values = _samples(style, shape, seed=i).astype(dtype)
            mode = MODES[i % 5]
            kind, options = KINDS[(i + len(style)) % len(KINDS)]
            for k, o in (("median", {}), (kind, options)):
                for omit, ignore_inf in ((False, False), (True, False), (True, True)):
                    with _core.Plan(shape, dtype, k, size, mode=[mode] * len(shape), cval=1.5, omit_nan=omit,
                                    ignore_inf=ignore_inf, **o) as plan:
                        assert plan.algorithm == "histogram"
                        actual = plan.run_host(values)
                    expected = oracle.window_filter(values, k, size, mode=mode, cval=1.5, omit_nan=omit,
                                                    ignore_inf=ignore_inf, parameter=o.get("parameter", 0),
                                                    q=o.get("percentile", 50.0))
                    np.testing.assert_array_equal(bits(actual), bits(expected),
                                                  err_msg=str((shape, size, k, omit, ignore_inf)))
    finally:
        _core.pin_kernel(None)
