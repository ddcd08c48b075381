"""Shared memory of the histogram kernel's tiles, as the library's host code
chooses them (a small program linked against it; no device is needed)."""

from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def tiles(tmp_path_factory):
    """tiles(windows): the chosen tile of each (D, H, W, kd, kh, kw, hole, double)."""
    from ndfiltrs_gb300 import _build

    library = _build.build()
    program = tmp_path_factory.mktemp("tiles") / "histogram_tiles"
    cuda = Path(_build.nvcc()).resolve().parent.parent / "include"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{cuda}", str(ROOT / "tests" / "histogram_tiles.cpp"), "-o",
                    str(program), str(library), f"-Wl,-rpath,{library.parent}"], check=True)

    def run(windows, sm_count=152):
        text = "\n".join(" ".join(str(int(v)) for v in w) for w in windows)
        lines = subprocess.run([str(program), str(sm_count)], input=text, capture_output=True, text=True, check=True).stdout.split("\n")
        return [tuple(int(v) for v in line.split()) for line in lines if line]

    return run


def _align16(n: int) -> int:
    return (n + 15) & ~15


def test_footprint_tiles_hold_their_axis_maps(tiles) -> None:
    """A footprint tile gathers its support through 64-bit offsets of the support's
    rows, planes and columns, which lie in the last region of shared memory, after
    the rank codes, the run lists and the decode table. The region must hold them;
    supports of two wide rows have little else there."""
    windows = [(d, h, w, kd, kh, kw, kw // 2, double)
               for d, h, w in ((1, 1, 5000), (1, 512, 16384), (3, 1, 5000))
               for kd, kh in ((1, 2), (2, 1), (1, 1), (1, 3))
               for kw in (*range(1990, 2010), *range(2100, 2150), *range(4960, 4980), *range(9990, 10010))
               for double in (0, 1)]
    seen = set()
    for (d, h, w, kd, kh, kw, hole, double), (tw, th, tz, sdec, in_smem, smem, entries) in zip(windows, tiles(windows)):
        if tw == 0:  # run lists too long for shared memory
            assert kw > 9000
            continue
        assert tz == 1 and not in_smem
        rows, columns = (th + kh - 1) * kd, tw + kw - 1
        support = rows * columns
        before = _align16(2 * support) + _align16(2 * entries) + (_align16(support * (8 if double else 4)) if sdec else 0)
        bitsets = 32 * 4 * ((support + 31) // 32)
        maps = 8 * (th + kh - 1 + kd + (columns if rows > 1 else 0))
        assert smem >= before + max(bitsets, maps, 17 * 256 * 4), (d, h, w, kd, kh, kw)
        if rows == 2:
            seen.add(columns % 16)
    assert seen >= {13, 14, 15, 0, 1}


def test_wide_boxes_find_a_tile(tiles) -> None:
    """Boxes of a few very wide rows: every box whose smallest tile fits the
    225 KB at six bytes a sample (rank codes and 32 segments' bit histograms; the
    run lists too of boxes deeper than a plane) has a tile, and the tile holds
    its codes, its places and the offsets of its rows."""
    budget = 225 * 1024
    windows, fits = [], 0
    for d, h, w in ((1, 1, 4000), (1, 3, 3000), (1, 600, 20000), (4, 5, 3000)):
        for kd, kh in ((1, 1), (1, 2), (1, 3), (1, 4), (1, 5), (1, 9), (2, 1), (3, 1), (2, 2)):
            if kd > 1 and d == 1:
                continue
            limit = 40000 // (kd * kh)
            windows += [(d, h, w, kd, kh, kw, -1, 0) for kw in range(limit // 4, limit, 97)]
    for (d, h, w, kd, kh, kw, _, _), (tw, th, tz, _, in_smem, smem, _) in zip(windows, tiles(windows)):
        smallest = kd * kh * (kw + 31)
        lists = 2 * (kd * kh * kw + 2 * kd * kw + 2 * kd * kh) if kd > 1 else 0
        if 2 * smallest + 16 + lists + 16 + max(17 * 256 * 4, 128 * ((smallest + 31) // 32)) > budget:
            continue
        fits += 1
        assert tw > 0, (d, h, w, kd, kh, kw)
        rows = (th + kh - 1) * (tz + kd - 1)
        support = rows * (tw + kw - 1)
        need = 8 * (th + kh - 1 + tz + kd - 1) + 2 * _align16(2 * (support + 64))
        assert need + (2 * support + 16 * 1024 if in_smem else 0) <= smem <= budget
    assert fits > 500


def test_flat_windows_share_their_supports(tiles) -> None:
    """The windows of test_gpu_histogram_wide.py that are walked along the rows have
    the tiles that give a warp several patches."""
    from tests.test_gpu_histogram_wide import SIDEWAYS

    for double in (0, 1):
        windows = [(1, *((1,) * (2 - len(shape)) + shape), 1, *((1,) * (2 - len(size)) + size), -1, double)
                   for shape, size, _ in SIDEWAYS]
        assert [t[:2] for t in tiles(windows)] == [tile for _, _, tile in SIDEWAYS]


def test_tiles_follow_the_sm_count(tiles) -> None:
    """Small arrays take tiles that leave no SM of the device without one."""
    windows = [(1, n, n, 1, k, k, -1, 0) for n in (300, 700, 1500) for k in (15, 33)]
    outputs = {sms: [t[0] * t[1] for t in tiles(windows, sms)] for sms in (19, 152)}
    assert outputs[19] != outputs[152]
    assert all(few >= many for few, many in zip(outputs[19], outputs[152]))


def test_deep_windows_sort_through_slots(tiles) -> None:
    """The cubes of test_gpu_histogram_deep.py have the tiles that they are there
    for, those of 64 x 512 x 512 among them, and slots in global memory."""
    from tests.test_gpu_histogram_deep import CUBES

    windows = [(*shape, *size, -1, double) for shape, size, double, _ in CUBES]
    for (_, _, _, tile), chosen in zip(CUBES, tiles(windows)):
        assert (chosen[:3], chosen[4]) == (tile, 0)
    assert tiles([(64, 512, 512, 9, 33, 33, -1, 0)])[0][:5] == (32, 20, 8, 0, 0)
