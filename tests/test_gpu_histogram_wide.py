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
