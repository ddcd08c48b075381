"""The mesh statistics' float32 decisions and 32-bit sort against the oracle, bit
for bit: mesh sizes around the sort's runs and the change of block size (4,096
and 16,384 samples), partial meshes, ranks 1 to 3, masks; samples with stars,
ties (spreads of zero, equal values on a limit), wide magnitudes and infinities."""

from __future__ import annotations

import numpy as np
import pytest

from tests.test_gpu_mesh import PHOTUTILS, _compare, _oracle_options

pytestmark = pytest.mark.gpu

SHAPES = [((130, 200), (64, 64)), ((70, 140), (65, 64)), ((260, 130), (128, 128)), ((140, 150), (129, 127)),
          ((9000,), (4097,)), ((300,), (1,)), ((33, 20), (3, 2)), ((9, 40, 50), (4, 17, 33)), ((64, 66), (2, 66))]


def _samples(style, shape, seed):
    rng = np.random.default_rng(seed)
    x = 500 + 22 * rng.normal(size=shape)
    if style == "stars":
        x = np.where(rng.random(shape) < 0.03, x + np.exp(rng.uniform(3, 11, shape)), x)
        x[rng.random(shape) < 0.02] = np.nan
    elif style == "ties":
        x = np.round(rng.normal(size=shape) * 2)
        x[rng.random(shape) < 0.6] = -0.0
    elif style == "wide":
        x = rng.normal(size=shape) * 10.0 ** rng.integers(-40, 38, shape)
        x[rng.random(shape) < 0.05] = np.inf
    return x.astype(np.float32)


@pytest.mark.parametrize("style", ("noise", "stars", "ties", "wide"))
def test_float32_meshes(gpu, oracle, style) -> None:
    for i, (shape, box) in enumerate(SHAPES):
        data = _samples(style, shape, seed=i)
        mask = np.random.default_rng(i).random(shape) < 0.1 if i % 2 else None
        for options in ({}, PHOTUTILS, {"estimator": "sigma_clip", "center": "mean", "statistic": "mean",
                                        "sigma_lower": 1.0, "sigma_upper": 2.5, "maxiters": None}):
            options = dict(options, min_valid_fraction=0.0)
            filter_size, oracle_options = _oracle_options(options)
            actual = gpu.mesh_background(data, box, mask=mask, **options)
            expected = oracle.mesh_background(data, box, filter_size, mask=mask, **oracle_options)
            _compare(actual, expected, (shape, box, options))


@pytest.mark.parametrize("shape,box", [((40, 700), (8, 5)), ((3, 5000), (3, 1)), ((19, 15000), (19, 1)), ((33, 64), (33, 64)),
                                       ((20, 257), (4, 300)), ((15, 14, 300), (5, 7, 16))])
def test_float32_maps(gpu, oracle, shape, box) -> None:
    """The spline's last axis: few and many nodes (staged or not), one node, remainders of its blocks,
    values large and small enough for float64."""
    rng = np.random.default_rng(len(shape))
    for scale in (1.0, 1e-30, 1e36):
        data = ((500 + 22 * rng.normal(size=shape)) * scale).astype(np.float32)
        actual = gpu.mesh_background(data, box, min_valid_fraction=0.0)
        expected = oracle.mesh_background(data, box, 3, min_valid_fraction=0.0, pearson=2.5)
        _compare(actual, expected, (shape, box, scale))
