"""Float32 moments whose integers fit 64-bit words, and tiles on either side of that
limit: powers of two of span, sums at the limit, zeros, subnormals, one class of
non-finite sample, against the exact window moments (2 ulp where the result is normal)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ("mean", "var", "std"))
@pytest.mark.parametrize("size", ((3, 3), (9, 31), (31, 31)))
def test_word_sums(gpu, oracle, kind, size) -> None:
    from ndfiltrs_gb300 import _core

    rng = np.random.default_rng(17)
    shape = (70, 97)
    whole = rng.integers(-1, 2, shape)
    images = {"zero": np.zeros(shape), "constant": np.full(shape, 3.0), "tiny": whole * 2.0**-149,
              "normal limit": (whole + 4) * 2.0**-126}
    for bits in (1, 8, 14, 19, 20, 21, 22, 24, 29, 30):  # magnitudes of the integers
        image = rng.integers(-(2**bits), 2**bits + 1, shape) * 2.0**-10
        image[::7, ::5] = 2.0**-10  # the lowest bit in every tile
        images[f"bits {bits}"] = image
    for scale in (-90, -49, -48, -26, 40):
        images[f"scale {scale}"] = (1e4 + rng.normal(size=shape)).astype(np.float32) * np.float64(2.0) ** scale
    for name, image in images.items():
        for ddof in (0, 1, 4) if kind != "mean" else (0,):
            values = image.astype(np.float32)
            if ddof != 4:
                values[rng.random(shape) < 0.05] = np.nan if ddof else -np.inf
            args = dict(omit_nan=True, ignore_inf=ddof != 1, min_count=1)
            with _core.Plan(shape, np.float32, kind, size, mode=["mirror"] * 2, parameter=ddof,
                            moments="fp32c", **args) as plan:
                assert plan.algorithm == "moments_slide"
                actual = plan.run_host(values)
            exact = oracle.exact_moments(values, kind, size, mode="mirror", ddof=ddof, **args)
            np.testing.assert_array_equal(np.isnan(actual), np.isnan(exact), err_msg=name)
            good = np.isfinite(exact) & (np.abs(exact) > np.finfo(np.float32).tiny)
            a, e = actual[good].astype(np.float64), exact[good].astype(np.float64)
            assert np.all(np.abs(a - e) <= 2 * np.spacing(np.abs(e).astype(np.float32))), (name, ddof)
            assert np.all(actual[exact == 0] == 0), (name, ddof)
