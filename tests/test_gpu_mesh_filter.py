"""The mesh median filter and the maps on the device against the oracle, bit for
bit: windows of one sample, even counts at edges, the largest that the device takes
and the first that it leaves, both edge rules and thresholds, invalid meshes, ranks 1
to 3, maps of which one is constant."""

from __future__ import annotations

import numpy as np
import pytest

from tests.test_gpu_mesh import _compare, _oracle_options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", (np.float32, np.float64))
@pytest.mark.parametrize("edge", ("shrink", "truncate"))
def test_filters(gpu, oracle, dtype, edge) -> None:
    cases = [((90, 70), (6, 5), f) for f in (1, (1, 3), 3, (5, 3), 11, (11, 13), (1, 123), (25, 1))]
    cases += [((300,), (4,), f) for f in (1, 3, 121, 123)] + [((20, 21, 22), (4, 5, 6), f) for f in (3, (3, 5, 7), (5, 5, 5))]
    cases += [((5, 6), (8, 8), 3), ((64, 3), (2, 3), (5, 3))]
    rng = np.random.default_rng(29)
    for shape, box, size in cases:
        data = (100 + 5 * rng.normal(size=shape)).astype(dtype)
        data[rng.random(shape) < 0.3] = np.nan
        flat = np.full(shape, 7.0, dtype)  # a spread of zero everywhere: a constant map of it
        for image, more in ((data, {"min_valid_fraction": 0.6}), (data, {"min_valid_fraction": 0.0}), (flat, {})):
            for rule in ({}, {"filter_threshold": 0.5}, {"filter_threshold": 100.0, "threshold_kind": "above"}):
                options = dict(more, filter_size=size, filter_edge=edge, **rule)
                filter_size, oracle_options = _oracle_options(dict(options))
                actual = gpu.mesh_background(image, box, **options)
                expected = oracle.mesh_background(image, box, filter_size, **oracle_options)
                _compare(actual, expected, (shape, box, options))
