"""The one-pass extrema kernel over segments of rows that are longer than tall
windows (arrays of one or two strips of 64 columns and many rows), and the two passes
that keep arrays of few columns, against the oracle, bit for bit. The oracle filters
the rows around the first and last outputs, the segments' borders and some between."""

from __future__ import annotations

import numpy as np
import pytest

from tests.conftest import bits

pytestmark = pytest.mark.gpu


def _check(oracle, shape, dtype, kind, size, mode, omit, seed, strips) -> None:
    """`strips`: the one-pass kernel, whose plan allocates nothing; the passes keep
    the array transposed."""
    import torch

    from ndfiltrs_gb300 import _core

    rng = np.random.default_rng(seed)
    values = (rng.integers(-1000, 1000, shape) * rng.random(shape)).astype(dtype)
    values[rng.random(shape) < 0.05] = dtype(-0.0)
    values[rng.random(shape) < 0.0005] = np.nan
    values[rng.random(shape) < 0.001] = np.inf
    _core.pin_kernel("passes")
    try:
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        with _core.Plan(shape, dtype, kind, size, mode=[mode] * 2, omit_nan=omit) as plan:
            assert plan.algorithm == "extrema_passes"
            taken = free - torch.cuda.mem_get_info()[0]
            assert taken == 0 if strips else taken >= values.nbytes
            actual = plan.run_host(values)
    finally:
        _core.pin_kernel(None)
    # Rows [a, b) of the result from the rows that their windows reach: whole where
    # the boundary is reached, else cut `kh` rows outside.
    height, kh = shape[0], size[0]
    for a in sorted({0, height // 3, height // 2 + 7, height - 400}):
        b = min(height, a + 400)
        low, high = max(0, a - kh), min(height, b + kh)
        expected = oracle.window_filter(values[low:high], kind, size, mode=mode, omit_nan=omit)[a - low:b - low]
        np.testing.assert_array_equal(bits(actual[a:b]), bits(expected), err_msg=str((shape, size, mode, omit, a)))


# 152 SMs take up to 16 warps each, so that the segments of an array of one strip
# are as long as H / 2432 rows: these heights leave each window twice (float64 2.5
# times) its rows.
@pytest.mark.parametrize("kind", ("min", "max"))
@pytest.mark.parametrize("dtype, size", ((np.float32, (31, 31)), (np.float32, (65, 65)), (np.float32, (97, 5)),
                                         (np.float32, (129, 2)), (np.float64, (31, 31)), (np.float64, (65, 3)),
                                         (np.float64, (97, 33))))
def test_tall_windows_match_oracle(gpu, oracle, kind, dtype, size) -> None:
    per_row = size[0] * 64 * np.dtype(dtype).itemsize
    warps = 4
    while warps > 1 and warps * per_row > 48 * 1024:
        warps //= 2
    resident = min(16, 227 * 1024 // (warps * per_row + 1024) * warps)
    rows = int(2.6 * size[0]) + 1
    height = 152 * resident * rows - 13
    for width, mode, omit in ((61, "reflect", True), (100, "mirror", False)):
        _check(oracle, (height // (1 + width // 65), width), dtype, kind, size, mode, omit, seed=size[0], strips=True)


@pytest.mark.parametrize("dtype", (np.float32, np.float64))
def test_few_columns_match_oracle(gpu, oracle, dtype) -> None:
    least = 16 if dtype == np.float32 else 33
    for i, (width, size) in enumerate(((1, (30, 1)), (2, (30, 1)), (5, (30, 1)), (15, (9, 3)), (16, (9, 3)), (32, (9, 3)),
                                       (33, (9, 3)), (3, (31, 5)))):
        _check(oracle, (600003, width), dtype, "min", size, ("nearest", "reflect", "constant")[i % 3], i % 2 == 0, seed=i,
               strips=width >= (2 if size[1] == 1 else least))
