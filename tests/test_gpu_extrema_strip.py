"""The one-pass extrema kernel (and, for arrays too short for it, the two passes)
against the oracle, bit for bit: window sides around each doubling (1 to 129 columns), strips of 64 columns and their remainders,
arrays smaller than the window, every mode, both dtypes and policies, with NaN,
infinities and signed zeros."""

from __future__ import annotations

import numpy as np
import pytest

from tests.conftest import bits

pytestmark = pytest.mark.gpu

MODES = ("reflect", "constant", "nearest", "mirror", "wrap")


@pytest.mark.parametrize("dtype", (np.float32, np.float64))
@pytest.mark.parametrize("kind", ("min", "max"))
def test_strips_match_oracle(gpu, oracle, kind, dtype) -> None:
    from ndfiltrs_gb300 import _core

    rng = np.random.default_rng(5)
    sides = (1, 2, 3, 4, 7, 8, 9, 15, 16, 17, 31, 32, 33, 47, 63, 64, 65, 95, 96, 97, 127, 128, 129)
    _core.pin_kernel("passes")
    try:
        for i, kw in enumerate(sides):
            kh = sides[(7 * i + 3) % len(sides)]
            for shape in ((40 + 9 * i, 64), (70, 63 + i), (3, 130), (150,), (3 * kh + 20, 70)):
                size = (kw,) if len(shape) == 1 else (kh, kw)
                values = (rng.integers(-3, 4, shape) * rng.random(shape)).astype(dtype)
                values[rng.random(shape) < 0.3] = dtype(-0.0)
                values[rng.random(shape) < 0.002] = np.nan
                values[rng.random(shape) < 0.05] = np.inf
                mode = MODES[(i + len(shape)) % 5]
                origin = tuple((-1) ** a * (k // 3) if k > 2 else 0 for a, k in enumerate(size))
                for omit, ignore_inf in ((False, False), (True, False), (True, True)):
                    with _core.Plan(shape, dtype, kind, size, origin=origin, mode=[mode] * len(shape), cval=0.5,
                                    omit_nan=omit, ignore_inf=ignore_inf) as plan:
                        assert plan.algorithm == "extrema_passes"
                        actual = plan.run_host(values)
                    expected = oracle.window_filter(values, kind, size, origin=origin, mode=mode, cval=0.5,
                                                    omit_nan=omit, ignore_inf=ignore_inf)
                    np.testing.assert_array_equal(bits(actual), bits(expected), err_msg=str((shape, size, mode)))
    finally:
        _core.pin_kernel(None)
