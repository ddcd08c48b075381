"""The histogram kernel over supports of a few very wide rows, whose axis maps
and rank codes fill shared memory, against the oracle, bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

from tests.conftest import bits

pytestmark = pytest.mark.gpu


def _samples(shape, dtype, seed):
    rng = np.random.default_rng(seed)
    values = rng.normal(size=shape)
    values[rng.random(shape) < 0.02] = np.nan
    values[rng.random(shape) < 0.02] = np.inf
    return values.astype(dtype)


def _check(oracle, shape, dtype, size, mode, footprint=None) -> None:
    from ndfiltrs_gb300 import _core

    values = _samples(shape, dtype, seed=size[-1])
    _core.pin_kernel("histogram")
    try:
        with _core.Plan(shape, dtype, "median", size, footprint=footprint, mode=[mode] * len(shape), cval=0.25,
                        omit_nan=True) as plan:
            assert plan.algorithm == "histogram"
            actual = plan.run_host(values)
    finally:
        _core.pin_kernel(None)
    expected = oracle.window_filter(values, "median", size, footprint=footprint, mode=mode, cval=0.25, omit_nan=True)
    np.testing.assert_array_equal(bits(actual), bits(expected), err_msg=str((shape, size, mode)))


@pytest.mark.parametrize("dtype", (np.float32, np.float64))
@pytest.mark.parametrize("width", (2110, 2111, 2112, 2126, 2127, 2128))
def test_wide_footprints_match_oracle(gpu, oracle, width, dtype) -> None:
    """Two support rows: SW = width + 127 around multiples of 16."""
    for shape, size, mode in (((1, 200), (2, width), "reflect"), ((2, 1, 150), (2, 1, width), "constant")):
        mask = np.ones(size, bool)
        mask.flat[width // 2] = False
        _check(oracle, shape, dtype, size, mode, mask)


@pytest.mark.parametrize("dtype", (np.float32, np.float64))
def test_wide_boxes_match_oracle(gpu, oracle, dtype) -> None:
    """Boxes whose columns have no table of offsets, and the widest that have one."""
    for shape, size, mode in (((3, 300), (2, 15000), "reflect"), ((2, 200), (2, 19000), "wrap"),
                              ((2, 200), (3, 12500), "constant"), ((40, 200), (4, 9000), "mirror"),
                              ((1, 500), (2, 14351), "nearest"), ((2, 3, 80), (2, 1, 15000), "reflect"),
                              ((2, 150), (2, 14350), "mirror"), ((2, 150), (2, 14320), "constant")):
        _check(oracle, shape, dtype, size, mode)


def test_wide_box_without_allocation(gpu, oracle) -> None:
    import ctypes

    import torch

    from tests.test_zz_no_alloc import KINDS, MODES, _entry_point

    lib, fn = _entry_point()
    shape, size = (3, 300), (2, 15000)
    values = _samples(shape, np.float32, seed=1)
    source = torch.from_numpy(values).cuda()
    target = torch.empty_like(source)
    rc = fn(source.data_ptr(), target.data_ptr(), 0, 2, (ctypes.c_uint64 * 2)(*shape), (ctypes.c_uint64 * 2)(*size),
            (ctypes.c_int64 * 2)(0, 0), (ctypes.c_int32 * 2)(MODES["reflect"], MODES["wrap"]), 0.0, KINDS["median"], 1, 0,
            1, 0, 50.0, torch.cuda.current_stream().cuda_stream)
    assert rc == 0, lib.ndf_last_error()
    torch.cuda.synchronize()
    expected = oracle.window_filter(values, "median", size, mode=["reflect", "wrap"], omit_nan=True)
    np.testing.assert_array_equal(bits(target.cpu().numpy()), bits(expected))


# Windows whose patches of outputs are walked along the rows, several to a warp:
# (shape, size, output tile).
SIDEWAYS = [((160000,), (2001,), (2048, 1)), ((160000,), (700,), (1024, 1)), ((100, 3000), (2, 1100), (1024, 1)),
            ((200, 1500), (3, 1500), (512, 2)), ((300, 1100), (1, 1500), (1024, 2)), ((400, 1030), (4, 1200), (512, 2))]


@pytest.mark.parametrize("style", ("noise", "slope", "steps", "sparse"))
@pytest.mark.parametrize("dtype", (np.float32, np.float64))
def test_flat_windows_match_oracle(gpu, oracle, dtype, style) -> None:
    from ndfiltrs_gb300 import _core

    for i, (shape, size, _) in enumerate(SIDEWAYS):
        rng = np.random.default_rng(i)
        x = np.arange(shape[-1])
        values = rng.normal(size=shape)
        if style == "slope":
            values = 0.01 * values + x
        elif style == "steps":
            values = np.where(x // 150 % 2 == 0, -1e3, 1e3) + np.round(values)
        elif style == "sparse":
            values[rng.random(shape) < 0.995] = np.nan
        values[rng.random(shape) < 0.0003] = np.inf
        values = values.astype(dtype)
        if style == "noise":
            values[..., 700:] = np.where(rng.random(values[..., 700:].shape) < 0.002, np.nan, values[..., 700:])
        rows = slice(0, 6) if len(shape) == 2 else slice(None)
        strip = values[:10] if len(shape) == 2 else values
        mode = ["reflect"] * (len(shape) - 1) + [("wrap", "constant", "mirror")[i % 3]]
        _core.pin_kernel("histogram")
        try:
            for kind, options, policies in (("median_histogram", {}, (True, False)),
                                            ("percentile", dict(percentile=97.0), (True,))):
                for omit in policies:
                    with _core.Plan(shape, dtype, kind, size, mode=mode, cval=0.5, omit_nan=omit, **options) as plan:
                        assert plan.algorithm == "histogram"
                        actual = plan.run_host(values)[rows]
                    expected = oracle.window_filter(strip, kind, size, mode=mode, cval=0.5, omit_nan=omit,
                                                    q=options.get("percentile", 50.0))[rows]
                    np.testing.assert_array_equal(bits(actual), bits(expected), err_msg=str((shape, size, kind, omit)))
        finally:
            _core.pin_kernel(None)
