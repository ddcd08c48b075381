"""Deep windows over cubes large enough for tiles of several patches of planes,
whose supports are sorted through slots in global memory, against the oracle, bit for
bit, over the whole cube."""

from __future__ import annotations

import numpy as np
import pytest

from tests.conftest import bits

pytestmark = pytest.mark.gpu

# (shape, size, float64, output tile): the tile and the slot of a 64 x 512 x 512 cube,
# planes beyond the last whole tile, one patch of planes to a tile.
CUBES = [((30, 256, 256), (9, 33, 33), 0, (32, 20, 8)), ((39, 199, 259), (9, 33, 33), 0, (32, 20, 8)),
         ((27, 256, 256), (9, 33, 33), 1, (32, 32, 4))]


@pytest.mark.parametrize("cube", range(len(CUBES)))
@pytest.mark.parametrize("omit", (True, False))
def test_deep_windows_match_oracle(gpu, oracle, cube, omit) -> None:
    from ndfiltrs_gb300 import _core

    shape, size, double, _ = CUBES[cube]
    rng = np.random.default_rng(cube)
    values = rng.normal(size=shape) + 0.05 * np.arange(shape[1])[:, None]
    if omit:
        values[rng.random(shape) < 0.02] = np.nan
        values[:, 40:60, 100:170] = np.nan  # windows of few samples
        values[rng.random(shape) < 0.01] = np.inf
    else:
        values[7, 100, 100] = np.nan
    values = values.astype(np.float64 if double else np.float32)
    mode = ("nearest", "reflect", "wrap")[cube]
    with _core.Plan(shape, values.dtype, "median_histogram", size, mode=[mode] * 3, omit_nan=omit,
                    ignore_inf=omit) as plan:
        assert plan.algorithm == "histogram"
        actual = plan.run_host(values)
    expected = oracle.window_filter(values, "median_histogram", size, mode=mode, omit_nan=omit, ignore_inf=omit)
    np.testing.assert_array_equal(bits(actual), bits(expected))
