"""The autotuner's choice file: a measured choice is written with its key and taken
from the file again; choices measured on other versions of the kernels (and those
whose key has no version) are not."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _algorithm() -> str:
    from ndfiltrs_gb300 import _core

    with _core.Plan((200, 200), np.float32, "min", (9, 9), omit_nan=True) as plan:
        return plan.algorithm


def test_choices_of_other_kernels_are_not_taken(gpu, tmp_path) -> None:
    import ndfiltrs_gb300 as nf

    path = tmp_path / "choices.txt"
    try:
        nf.set_autotune(0, "")
        usual = _algorithm()
        assert usual == "extrema_passes"
        nf.set_autotune(2, str(path))
        _algorithm()
        key = path.read_text().split()[0]
        assert nf.autotune_entries() == 1
        version, _, rest = key.partition("/")

        def with_file(key):
            path.write_text(f"{key} extrema 0 0 0.01\n")
            nf.set_autotune(1, str(path))
            return nf.autotune_entries(), _algorithm()

        assert with_file(key) == (1, "extrema_tile")
        assert rest.startswith("sm")
        for stale in (rest, "k1/" + rest, version + "0/" + rest):
            assert with_file(stale) == (0, usual)
    finally:
        nf.set_autotune(0, "")


def test_box_tiles_follow_the_array(gpu) -> None:
    """The histogram's tile of a box depends on the array's size, which a choice's
    key does not hold: boxes have one candidate, nothing to measure, and footprints
    several."""
    import ndfiltrs_gb300 as nf
    from ndfiltrs_gb300 import _core

    disk = np.add.outer(np.arange(-9, 10) ** 2, np.arange(-9, 10) ** 2) <= 81
    try:
        nf.set_autotune(2, "")
        for footprint, entries in ((None, 0), (disk, 1)):
            with _core.Plan((200, 200), np.float32, "median", (19, 19), footprint=footprint, omit_nan=True) as plan:
                assert plan.algorithm == "histogram"
            assert nf.autotune_entries() == entries
    finally:
        nf.set_autotune(0, "")
