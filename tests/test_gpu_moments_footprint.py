"""Float32 moments of footprints whose taps are one word or two: whole tiles of
finite samples, one and several classes of non-finite ones, 1,023 and 1,024 taps (the
limit of the class fields), deviations on either side of 31 bits, 3-D windows, against
the exact window moments (2 ulp where the result is normal)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _taps(shape, count, rng):
    flat = np.zeros(int(np.prod(shape)), dtype=bool)
    flat[rng.choice(flat.size, size=count, replace=False)] = True
    return flat.reshape(shape)


@pytest.mark.parametrize("kind", ("mean", "var", "std"))
def test_footprints(gpu, oracle, kind) -> None:
    from ndfiltrs_gb300 import _core

    rng = np.random.default_rng(41)
    cases = [((40, 75), _taps((5, 7), 12, rng)), ((40, 75), _taps((13, 13), 113, rng)), ((70, 66), _taps((33, 33), 1023, rng)),
             ((70, 66), _taps((33, 33), 1024, rng)), ((6, 20, 40), _taps((3, 5, 5), 40, rng)), ((6, 20, 40), _taps((3, 3, 3), 27, rng))]
    for shape, taps in cases:
        level = 1e4 + rng.normal(size=shape)
        whole = rng.integers(-(2**22), 2**22, shape) * 2.0**-8
        wide = rng.integers(-(2**30), 2**30, shape).astype(np.float64)
        for name, base in (("level", level), ("whole", whole), ("wide", wide), ("tiny", level * 2.0**-100)):
            for classes in ((), (np.nan,), (np.nan, np.inf, -np.inf)):
                values = base.astype(np.float32)
                for c in classes:
                    values[rng.random(shape) < 0.03] = c
                for ddof, omit, drop in ((0, True, True), (1, True, False), (2, False, False)):
                    args = dict(omit_nan=omit, ignore_inf=drop, min_count=1)
                    ddof = 0 if kind == "mean" else ddof
                    with _core.Plan(shape, np.float32, kind, taps.shape, footprint=taps, mode=["reflect"] * len(shape),
                                    parameter=ddof, moments="fp32c", **args) as plan:
                        actual = plan.run_host(values)
                    exact = oracle.exact_moments(values, kind, taps.shape, footprint=taps, mode="reflect", ddof=ddof, **args)
                    context = (shape, int(taps.sum()), name, classes, ddof, omit)
                    np.testing.assert_array_equal(np.isnan(actual), np.isnan(exact), err_msg=str(context))
                    np.testing.assert_array_equal(actual[np.isinf(exact)], exact[np.isinf(exact)].astype(np.float32))
                    good = np.isfinite(exact) & (np.abs(exact) > np.finfo(np.float32).tiny)
                    a, e = actual[good].astype(np.float64), exact[good]
                    assert np.all(np.abs(a - e) <= 2 * np.spacing(np.abs(e).astype(np.float32))), context
