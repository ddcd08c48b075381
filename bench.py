"""Benchmark of the GB300 windowed-statistics path (one JSON line on stdout).

Default workload: ``nanmedian_filter(method="sortnet")`` with a 5x5 box on
one 4096x4096 float32 image (the robust-statistics image: background
1000 + 50*x/4096, Normal(0, 10) noise, 0.2% outliers Uniform(2000, 60000),
0.5% NaN, 0.1% +inf; seeded, synthetic). One step filters one image.

* ``value``: Mpix/s with the input already in HBM (device pointers through
  the C-ABI plan), timed with CUDA events on the launching stream. Inputs
  rotate over ``max(4, ceil(3 x 129 MiB / image bytes))`` device buffers
  (seven 67 MB images for the default workload, 470 MB > 3 x 129 MB L2), so
  no step reads an input that the previous steps left in L2.
* ``e2e``: the same metric through the C-ABI host-buffer entry point
  (``ndf_plan_run_host``): pinned host input -> device -> kernel -> pinned
  host output, synchronized every step.
* ``roofline``: algorithmic HBM bytes per launch (4 B read + 4 B written per
  pixel) / the launch's average duration, against the measured HBM copy
  bandwidth; selection is instruction-bound, so this fraction is low by
  design (see profiles/ for issue-slot utilization).
* ``cpu_baseline``: the CPU oracle (a restatement of the reference's Rust
  sortnet path, the reference itself cannot be built here) on a bounded
  strip of the same image with all host threads.

``--impl reference`` times that CPU path alone as the reference arm.
Under torchrun with N > 1 every rank filters its own image (independent
replicas, weak scaling, no collective on the data path).
"""

from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))

METRIC = "nanmedian Mpix/s on 1 GB300 (plain vs batched); nanstd max rel err vs FP64"


# ---------------------------------------------------------------------------
# Synthetic inputs (shapes and distributions of the benchmark configurations).

def robust_image(n: int = 4096, seed: int = 2) -> np.ndarray:
    rng = np.random.default_rng(seed)
    x = np.arange(n, dtype=np.float64)
    image = (1000.0 + 50.0 * x / n)[None, :] + rng.normal(0.0, 10.0, size=(n, n))
    outliers = rng.random((n, n)) < 0.002
    image[outliers] = rng.uniform(2000.0, 60000.0, size=int(outliers.sum()))
    image[rng.random((n, n)) < 0.005] = np.nan
    image[rng.random((n, n)) < 0.001] = np.inf
    return image.astype(np.float32)


def gaussian_image(n: int = 2048, seed: int = 1) -> np.ndarray:
    rng = np.random.default_rng(seed)
    image = rng.normal(1000.0, 10.0, size=(n, n))
    image[rng.random((n, n)) < 0.01] = np.nan
    return image.astype(np.float32)


def sky_image(n: int = 8192, seed: int = 3, dtype=np.float32) -> np.ndarray:
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:n, 0:n].astype(np.float64)
    sky = 500.0 + 0.01 * x - 0.005 * y
    image = sky + rng.normal(size=(n, n)) * np.sqrt(sky)
    count = 20000 if n >= 8192 else max(1, int(20000 * (n / 8192) ** 2))
    cy, cx = rng.uniform(0, n, size=count), rng.uniform(0, n, size=count)
    sigma = rng.uniform(1.5, 3.0, size=count)
    peak = np.exp(rng.uniform(np.log(50.0), np.log(50000.0), size=count))
    for k in range(count):
        r = int(np.ceil(4 * sigma[k]))
        y0, y1 = max(0, int(cy[k]) - r), min(n, int(cy[k]) + r + 1)
        x0, x1 = max(0, int(cx[k]) - r), min(n, int(cx[k]) + r + 1)
        if y0 >= y1 or x0 >= x1:
            continue
        yy, xx = np.mgrid[y0:y1, x0:x1]
        image[y0:y1, x0:x1] += peak[k] * np.exp(-0.5 * ((yy - cy[k]) ** 2 + (xx - cx[k]) ** 2) / sigma[k] ** 2)
    image[:, rng.choice(n, size=8, replace=False)] = np.nan
    return image.astype(dtype)


def precision_image(n: int = 4096, seed: int = 4, dtype=np.float32) -> np.ndarray:
    rng = np.random.default_rng(seed)
    image = 1e4 + rng.normal(size=(n, n))
    image[rng.random((n, n)) < 0.01] = np.nan
    return image.astype(dtype)


def cube_image(seed: int = 2, shape=(64, 1024, 1024)) -> np.ndarray:
    """64 x 1024 x 1024 float32 cube with the robust image's distribution."""
    rng = np.random.default_rng(seed)
    x = np.arange(shape[2], dtype=np.float32)
    image = (np.float32(1000) + np.float32(50) * x / np.float32(shape[2]))[None, None, :] + \
        rng.standard_normal(shape, dtype=np.float32) * np.float32(10)
    outliers = rng.random(shape, dtype=np.float32) < 0.002
    image[outliers] = rng.uniform(2000.0, 60000.0, size=int(outliers.sum())).astype(np.float32)
    image[rng.random(shape, dtype=np.float32) < 0.005] = np.nan
    image[rng.random(shape, dtype=np.float32) < 0.001] = np.inf
    return image


def _ring() -> np.ndarray:
    from ndfiltrs_gb300 import kernels

    return kernels.ring(4, 6, 2) != 0


def _tophat() -> np.ndarray:
    from ndfiltrs_gb300 import kernels

    return kernels.tophat(1, 2) != 0


class Workload:
    """One benchmark configuration: an image generator and the filter."""

    def __init__(self, gen, kind, size, mode, omit=True, ignore_inf=False, min_count=1, parameter=0,
                 q=50.0, footprint=None, origin=None, robust=None):
        self.gen, self.kind, self.size, self.mode = gen, kind, size, mode
        self.omit, self.ignore_inf, self.min_count, self.parameter = omit, ignore_inf, min_count, parameter
        self.q, self.footprint_fn, self.origin = q, footprint, origin
        self.robust = robust  # estimator options of the robust kinds

    def footprint(self):
        return self.footprint_fn() if self.footprint_fn is not None else None

    def window(self):
        fp = self.footprint()
        return tuple(fp.shape) if fp is not None else tuple(self.size)


WORKLOADS = {
    # Robust-statistics image, 4096 x 4096 float32 (sortnet / box kernels).
    "nanmedian_sortnet_5x5_4096_f32": Workload(lambda: robust_image(4096), "median_network", (5, 5), "reflect"),
    "nanmedian_sortnet_7x7_4096_f32": Workload(lambda: robust_image(4096), "median_network", (7, 7), "reflect"),
    "rank2_5x5_4096_f32": Workload(lambda: robust_image(4096), "rank", (5, 5), "reflect", omit=False, parameter=2),
    "nanpercentile84_5x5_4096_f32": Workload(lambda: robust_image(4096), "percentile", (5, 5), "reflect", q=84.0),
    "nanmedian_ring_4_6_4096_f32": Workload(lambda: robust_image(4096), "median_network", None, "reflect",
                                            footprint=_ring),
    "nanmedian_tophat1_4096_f32": Workload(lambda: robust_image(4096), "median_network", None, "constant",
                                           footprint=_tophat, origin=(1, -1)),
    "nanmedian_sortnet_3x5x5_cube_f32": Workload(cube_image, "median_network", (3, 5, 5), "reflect"),
    # 3-D sliding histogram: a (9, 33, 33) window (9,801 taps) on a 64 x 512 x 512 cube.
    "nanmedian_hist_9x33x33_cube512_f32": Workload(lambda: cube_image(shape=(64, 512, 512)), "median_histogram",
                                                   (9, 33, 33), "nearest"),
    # Gaussian image, 2048 x 2048 float32, direct 3 x 3.
    "nanmedian_direct_3x3_2048_f32": Workload(lambda: gaussian_image(2048), "median", (3, 3), "reflect"),
    # Sky image, histogram method, mode nearest.
    "nanmedian_hist_65x65_4096_f32": Workload(lambda: sky_image(4096), "median_histogram", (65, 65), "nearest"),
    # The mixed batch's largest boxes (13 x 13 and 15 x 15 run on the sliding histogram).
    "nanmedian_hist_13x13_4096_f32": Workload(lambda: sky_image(4096), "median_histogram", (13, 13), "nearest"),
    "nanmedian_hist_65x65_8192_f32": Workload(lambda: sky_image(8192), "median_histogram", (65, 65), "nearest"),
    "nanmedian_hist_129x129_8192_f32": Workload(lambda: sky_image(8192), "median_histogram", (129, 129), "nearest"),
    "nanmedian_hist_65x65_8192_f64": Workload(lambda: sky_image(8192, dtype=np.float64), "median_histogram",
                                              (65, 65), "nearest"),
    "nanmedian_hist_129x129_8192_f64": Workload(lambda: sky_image(8192, dtype=np.float64), "median_histogram",
                                                (129, 129), "nearest"),
    # Precision image, nanstd (FP32-compensated moments).
    "nanstd_31x31_4096_f32": Workload(lambda: precision_image(4096), "std", (31, 31), "reflect", ignore_inf=True,
                                      min_count=5, parameter=1),
    "nanstd_7x51_4096_f32": Workload(lambda: precision_image(4096), "std", (7, 51), "reflect", ignore_inf=True,
                                     min_count=5, parameter=1),
    "nanstd_31x31_4096_f64": Workload(lambda: precision_image(4096, dtype=np.float64), "std", (31, 31), "reflect",
                                      ignore_inf=True, min_count=5, parameter=1),
    # Separable rectangular extrema (van Herk / Gil-Werman).
    "nanmin_31x31_4096_f32": Workload(lambda: robust_image(4096), "min", (31, 31), "reflect"),
    "nanmax_65x65_8192_f32": Workload(lambda: sky_image(8192), "max", (65, 65), "nearest"),
    # Exact rolling means (method="boxcar"), correctly rounded.
    "nanmean_boxcar_31x31_4096_f32": Workload(lambda: precision_image(4096), "mean_rolling", (31, 31), "reflect",
                                              ignore_inf=True, min_count=5),
    "nanmean_boxcar_129x129_8192_f32": Workload(lambda: sky_image(8192), "mean_rolling", (129, 129), "nearest"),
    "nanmean_boxcar_31x31_4096_f64": Workload(lambda: precision_image(4096, dtype=np.float64), "mean_rolling",
                                              (31, 31), "reflect", ignore_inf=True, min_count=5),
    # Robust family (per-window float64 estimators).
    "nanmad_5x5_4096_f32": Workload(lambda: robust_image(4096), "mad", (5, 5), "reflect",
                                    robust=dict(parameter=1.0)),
    "sigma_clip_mode_7x7_2048_f32": Workload(lambda: robust_image(2048), "sigma_mode", (7, 7), "reflect",
                                             robust=dict(sigma_lower=3.0, sigma_upper=3.0, maxiters=None,
                                                         center="median", spread="std", estimator="sex",
                                                         pearson=2.5)),
    "biweight_location_7x7_2048_f32": Workload(lambda: robust_image(2048), "biweight_location", (7, 7),
                                               "reflect", robust=dict(parameter=6.0)),
}
ROBUST_KINDS = ("mad", "mode", "biweight_location", "biweight_scale", "sigma_mean", "sigma_median",
                "sigma_mode")
DEFAULT_WORKLOAD = "nanmedian_sortnet_5x5_4096_f32"

# DRAM bytes (read + write) per launch of the workload's kernel, from one ncu
# capture each (profiles/<kernel>_<workload>.md). Writes that are still in L2
# when the kernel ends are not counted there.
MEASURED_TRAFFIC = {
    "nanmedian_sortnet_5x5_4096_f32": (67.182592e6 + 29.531392e6, "profiles/tile_box_kernel_nanmedian_sortnet_5x5_4096_f32.md"),
    "nanmedian_hist_65x65_4096_f32": (67.946240e6 + 39.831552e6, "profiles/histogram_kernel_nanmedian_hist_65x65_4096_f32.md"),
    "nanmedian_ring_4_6_4096_f32": (67.191808e6 + 28.039424e6, "profiles/rank_network_kernel_nanmedian_ring_4_6_4096_f32.md"),
    "nanstd_31x31_4096_f32": (67.203072e6 + 30.213632e6, "profiles/moments_slide_kernel_nanstd_31x31_4096_f32.md"),
    "nanmin_31x31_4096_f32": (84.810240e6 + 23.049728e6, "profiles/extrema_strip_kernel_nanmin_31x31_4096_f32.md"),
    "nanmad_5x5_4096_f32": (67.206400e6 + 31.348736e6, "profiles/robust_tile_kernel_nanmad_5x5_4096_f32.md"),
}


# Warp instructions one filter call issues (all its launches), from the
# workload's ncu capture: the issue-rate roofline of the selection and
# integer kernels, whose bound is the instruction issue rather than HBM.
MEASURED_INSTRUCTIONS = {
    "nanmedian_sortnet_5x5_4096_f32": (211559951, "profiles/tile_box_kernel_nanmedian_sortnet_5x5_4096_f32.md"),
    "nanmedian_hist_65x65_4096_f32": (2193752494, "profiles/histogram_kernel_nanmedian_hist_65x65_4096_f32.md"),
    "nanmedian_ring_4_6_4096_f32": (875186480, "profiles/rank_network_kernel_nanmedian_ring_4_6_4096_f32.md"),
    "nanstd_31x31_4096_f32": (344461279, "profiles/moments_slide_kernel_nanstd_31x31_4096_f32.md"),
    "nanmin_31x31_4096_f32": (80728736, "profiles/extrema_strip_kernel_nanmin_31x31_4096_f32.md"),
    "nanmean_boxcar_31x31_4096_f32": (389130095, "profiles/boxcar_band_kernel_nanmean_boxcar_31x31_4096_f32.md"),
    "nanmad_5x5_4096_f32": (593685816, "profiles/robust_tile_kernel_nanmad_5x5_4096_f32.md"),
}


def issue_roofline(workload: str, ms_per_step: float, sm_count: int, sm_mhz: float | None) -> dict | None:
    """Warp instructions per second against the SMs' issue peak (four
    schedulers per SM, one warp instruction each per clock, at the sampled
    SM clock)."""
    known = MEASURED_INSTRUCTIONS.get(workload)
    if known is None or not sm_mhz:
        return None
    achieved = known[0] / (ms_per_step / 1e3) / 1e9
    peak = sm_count * 4 * sm_mhz * 1e6 / 1e9
    return {"achieved": round(achieved, 1), "peak": round(peak, 1), "unit": "G warp instructions/s",
            "frac": round(achieved / peak, 4), "instructions_per_call": int(known[0]), "source": known[1]}


# Kernels of this library one filter call launches, where it is more than one: the
# band and tiled exact means add a wider pass and the direct pass for bands or
# tiles their words cannot hold, the MAD and sigma clipping the pass that
# finishes the windows their tile kernel marks.
LAUNCHES_PER_CALL = {"boxcar_band": 3, "boxcar_tile": 2, "robust mad": 2, "robust sigma_mode": 2}


def oracle_kind(kind: str) -> str:
    return kind


# ---------------------------------------------------------------------------
# Clock sampling during the timed region.

class ClockSampler:
    """SM clock and clock-event reasons during the timed region, read (only
    read) through NVML from the driver's libnvidia-ml every 2 ms in a
    background thread plus at the region's start and end; falls back to
    polling nvidia-smi when NVML cannot be loaded."""

    REASONS = {0x4: "sw_power_cap", 0x8: "hw_slowdown", 0x20: "sw_thermal_slowdown",
               0x40: "hw_thermal_slowdown", 0x80: "hw_power_brake_slowdown"}

    def __init__(self, device: int) -> None:
        self.device = device
        self.samples: list[tuple[float, int]] = []
        self.max_mhz = None
        self.source = "nvml"
        self._stop = None
        self._thread = None
        self._nvml = None
        self._handle = None
        self._smi = None

    def _open_nvml(self) -> bool:
        import ctypes

        try:
            lib = ctypes.CDLL("libnvidia-ml.so.1")
            if lib.nvmlInit_v2() != 0:
                return False
            handle = ctypes.c_void_p()
            ok = False
            try:
                import torch

                uuid = str(torch.cuda.get_device_properties(self.device).uuid)
                ok = lib.nvmlDeviceGetHandleByUUID(("GPU-" + uuid).encode(), ctypes.byref(handle)) == 0
            except Exception:
                ok = False
            if not ok and lib.nvmlDeviceGetHandleByIndex_v2(self.device, ctypes.byref(handle)) != 0:
                return False
            self._nvml, self._handle = lib, handle
            maxc = ctypes.c_uint(0)
            if lib.nvmlDeviceGetMaxClockInfo(handle, 1, ctypes.byref(maxc)) == 0:
                self.max_mhz = float(maxc.value)
            return True
        except OSError:
            return False

    def _sample(self) -> None:
        import ctypes

        clock, reasons = ctypes.c_uint(0), ctypes.c_ulonglong(0)
        if self._nvml.nvmlDeviceGetClockInfo(self._handle, 1, ctypes.byref(clock)) != 0:
            return
        getter = getattr(self._nvml, "nvmlDeviceGetCurrentClocksEventReasons", None) or \
            self._nvml.nvmlDeviceGetCurrentClocksThrottleReasons
        getter(self._handle, ctypes.byref(reasons))
        self.samples.append((float(clock.value), int(reasons.value)))

    def __enter__(self):
        import threading

        if self._open_nvml():
            self._sample()
            self._stop = threading.Event()

            def loop() -> None:
                while not self._stop.wait(0.002):
                    self._sample()

            self._thread = threading.Thread(target=loop, daemon=True)
            self._thread.start()
        else:
            self.source = "nvidia-smi"
            try:
                self._file = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
                self._smi = subprocess.Popen(
                    ["nvidia-smi", "--query-gpu=clocks.sm,clocks.max.sm,clocks_event_reasons.active",
                     "--format=csv,noheader,nounits", "-lms", "200", "-i", str(self.device)],
                    stdout=self._file, stderr=subprocess.DEVNULL)
            except (OSError, FileNotFoundError):
                self._smi = None
        return self

    def __exit__(self, *exc) -> None:
        if self._thread is not None:
            self._stop.set()
            self._thread.join(timeout=2)
            self._sample()
        if self._smi is not None:
            self._smi.terminate()
            try:
                self._smi.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self._smi.kill()
            self._file.flush()
            for line in Path(self._file.name).read_text().strip().splitlines():
                parts = [p.strip() for p in line.split(",")]
                try:
                    self.samples.append((float(parts[0]), int(parts[2], 16)))
                    self.max_mhz = float(parts[1])
                except (ValueError, IndexError):
                    continue
            os.unlink(self._file.name)

    def summary(self) -> dict:
        if not self.samples:
            return {"sm_mhz": None, "sm_max_mhz": self.max_mhz, "reasons": ["no clock samples"],
                    "samples": 0, "source": self.source}
        reasons = sorted({name for _, bits in self.samples for mask, name in self.REASONS.items() if bits & mask})
        return {"sm_mhz": statistics.median(mhz for mhz, _ in self.samples), "sm_max_mhz": self.max_mhz,
                "reasons": reasons, "samples": len(self.samples), "source": self.source}


# ---------------------------------------------------------------------------
# Replicas across ranks: every rank filters its own image; the job's time is
# the slowest rank's and its throughput counts every rank's pixels.

def max_over_ranks(value: float, dist, device, barrier: bool = True) -> float:
    """The maximum of `value` over all ranks (the value itself without a
    process group), after a barrier."""
    if dist is None:
        return float(value)
    import torch

    if barrier:
        dist.barrier()
    t = torch.tensor([float(value)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def replica_throughput(world: int, pixels: int, steps: int, seconds: float) -> float:
    """Whole-job Mpix/s: all ranks' pixels over the slowest rank's time."""
    return world * pixels * steps / seconds / 1e6


def measured_peak_hbm() -> tuple[float, str]:
    path = ROOT / "MEASURED_PEAKS.json"
    if path.exists():
        try:
            return float(json.loads(path.read_text())["hbm_gbs"]), "measured"
        except (KeyError, ValueError):
            pass
    return 6800.0, "fallback"


# ---------------------------------------------------------------------------
# CPU baseline (the oracle on a bounded strip of the same image).

def cpu_baseline(image: np.ndarray, spec, budget_s: float = 3.0, threads: int | None = None) -> dict:
    from oracle import oracle

    oracle.build()
    threads = threads or (os.cpu_count() or 1)
    per_row = image[0].size
    first = 16 if image.ndim < 3 else 2

    def run(rows: int) -> float:
        strip = np.ascontiguousarray(image[:rows])
        start = time.perf_counter()
        oracle_filter(oracle, spec, strip, threads)
        return time.perf_counter() - start

    # Grow the slab until one call takes about a third of the budget (fixed
    # per-call costs make a short first call a poor predictor).
    rows = first
    elapsed = run(rows)
    while rows < image.shape[0] and elapsed < budget_s / 3:
        grow = int(rows * (budget_s / 3) / max(elapsed, 1e-6))
        rows = int(min(image.shape[0], max(2 * rows, grow)))
        elapsed = run(rows)
    times = [elapsed] + [run(rows) for _ in range(2)]
    seconds = statistics.median(times)
    mpix = rows * per_row / seconds / 1e6
    sample_shape = "x".join(str(v) for v in (rows,) + image.shape[1:])
    separable = spec.footprint() is None and spec.kind in ("min", "max", "mean_rolling")
    algorithm = f"{spec.kind}, separable axis passes" if separable else spec.kind
    return {
        "value": round(mpix, 3),
        "unit": "Mpix/s",
        "cores": threads,
        "kind": "port",
        "rows": rows,
        "sample": f"{sample_shape} leading slab of the same image, median of 3 calls, "
                  f"oracle restatement of the reference algorithm ({algorithm}), {threads} threads",
    }


def oracle_filter(oracle, spec, array, threads=None):
    if spec.kind in ROBUST_KINDS:
        clip = spec.kind.startswith("sigma")
        return oracle.robust_filter(array, spec.kind, spec.window(), footprint=spec.footprint(),
                                    origin=spec.origin if spec.origin is not None else 0, mode=spec.mode,
                                    omit_nan=spec.omit or clip, ignore_inf=spec.ignore_inf or clip,
                                    min_count=spec.min_count, threads=threads, **(spec.robust or {}))
    return oracle.window_filter(array, spec.kind, spec.window(), footprint=spec.footprint(),
                                origin=spec.origin if spec.origin is not None else 0, mode=spec.mode, omit_nan=spec.omit,
                                ignore_inf=spec.ignore_inf, min_count=spec.min_count,
                                parameter=spec.parameter, q=spec.q, threads=threads)


# ---------------------------------------------------------------------------
# Batched mixed workload: many float32 images of uneven sizes.

def mixed_batch(count: int = 512, seed: int = 5, lo: int = 256, hi: int = 4096):
    """Per image: sides log-uniform in [lo, hi] per axis, 1% NaN, 0.2%
    outliers; window in {3, 5, ..., 15}; footprint box / tophat / ring(r, r+2);
    filter nanmedian / nanpercentile 84 / nanstd."""
    from ndfiltrs_gb300 import kernels

    rng = np.random.default_rng(seed)
    specs, images = [], []
    for i in range(count):
        h = int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))
        w = int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))
        image = rng.standard_normal((h, w), dtype=np.float32) * np.float32(10) + np.float32(1000)
        image[rng.random((h, w), dtype=np.float32) < 0.01] = np.nan
        outliers = rng.random((h, w), dtype=np.float32) < 0.002
        image[outliers] = rng.uniform(2000.0, 60000.0, size=int(outliers.sum())).astype(np.float32)
        window = int(rng.choice(np.arange(3, 16, 2)))
        footprint_kind = rng.choice(["box", "tophat", "ring"])
        footprint = None
        if footprint_kind == "tophat":
            footprint = kernels.tophat(window // 2, 2) != 0
        elif footprint_kind == "ring":
            outer = max(window // 2, 2)
            footprint = kernels.ring(outer - 2, outer, 2) != 0
        filt = rng.choice(["nanmedian", "percentile", "nanstd"])
        kind = {"nanmedian": "median", "percentile": "percentile", "nanstd": "std"}[str(filt)]
        specs.append(dict(shape=(h, w), kind=kind, size=(window, window), footprint=footprint,
                          omit_nan=True, ignore_inf=kind == "std", min_count=1,
                          parameter=1 if kind == "std" else 0, percentile=84.0, mode="reflect"))
        images.append(image)
    return specs, images


def public_call(nf, spec, image):
    """One image through the public per-call API (what a caller of the
    reference loops over)."""
    footprint = spec["footprint"]
    size = None if footprint is not None else spec["size"]
    if spec["kind"] == "median":
        return nf.nanmedian_filter(image, size, footprint=footprint, mode=spec["mode"])
    if spec["kind"] == "percentile":
        return nf.nanpercentile_filter(image, spec["percentile"], size, footprint=footprint, mode=spec["mode"])
    return nf.nanstd_filter(image, size, footprint=footprint, mode=spec["mode"], ddof=spec["parameter"],
                            ignore_inf=spec["ignore_inf"])


def batch_comparison(args, public_loop: bool = True) -> dict:
    """The mixed-size batch (512 float32 images, window 3..15, box / tophat /
    ring, nanmedian / nanpercentile 84 / nanstd) through one batched launch
    set against the plain per-call GPU path. Device-resident, CUDA events on
    the launching stream:

    * ``plain_per_call``: per image, create the plan (``ndf_plan_create``:
      validation, window tables, kernel choice, device buffers), run it on
      the device buffers and destroy it -- what a caller looping the
      one-call API over images of different shapes and windows pays;
    * ``plain_prebuilt``: the same loop over plans built beforehand (the
      kernels alone, launched one image after another);
    * ``batched``: ``ndf_batch_run`` (persistent family launches replayed from
      a CUDA graph).

    End to end (host arrays in, host arrays out): one ``Batch.run_host`` call
    against the public per-call API in a loop. Outputs are compared bit for
    bit."""
    import torch

    import ndfiltrs_gb300 as nf

    specs, images = mixed_batch(args.batch_images)
    pixels = int(sum(im.size for im in images))
    device = torch.device("cuda", 0)
    d_in = [torch.from_numpy(im).to(device) for im in images]
    d_plain = [torch.empty_like(t) for t in d_in]
    d_batch = [torch.empty_like(t) for t in d_in]
    stream = torch.cuda.Stream(device)
    handle = stream.cuda_stream
    # The batch measures the kernel choices of its (dtype, window, footprint
    # class) keys first; the per-image plans below then use the same choices.
    t0 = time.perf_counter()
    batch = nf.Batch(specs)
    batch_create_s = time.perf_counter() - t0

    def make_plan(spec):
        kw = dict(footprint=spec["footprint"], omit_nan=True, ignore_inf=spec["ignore_inf"],
                  min_count=1, parameter=spec["parameter"], percentile=84.0, mode=["reflect"] * 2)
        size = spec["footprint"].shape if spec["footprint"] is not None else spec["size"]
        return nf.Plan(spec["shape"], np.float32, spec["kind"], size, **kw)

    plans = [make_plan(spec) for spec in specs]
    in_ptrs = [t.data_ptr() for t in d_in]
    out_ptrs = [t.data_ptr() for t in d_batch]

    def percall_step() -> None:
        for spec, src, dst in zip(specs, d_in, d_plain):
            plan = make_plan(spec)
            plan.run_device(src.data_ptr(), dst.data_ptr(), handle)
            plan.close()

    def prebuilt_step() -> None:
        for plan, src, dst in zip(plans, d_in, d_plain):
            plan.run_device(src.data_ptr(), dst.data_ptr(), handle)

    def batch_step() -> None:
        batch.run_device(in_ptrs, out_ptrs, handle)

    def timed(fn, steps, warmup):
        for _ in range(warmup):
            fn()
        torch.cuda.synchronize()
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0 = time.perf_counter()
        start.record(stream)
        for _ in range(steps):
            fn()
        end.record(stream)
        torch.cuda.synchronize()
        return start.elapsed_time(end) / steps, (time.perf_counter() - t0) / steps * 1e3

    def wall(fn, steps, warmup=1):
        for _ in range(warmup):
            fn()
        t0 = time.perf_counter()
        for _ in range(steps):
            result = fn()
        return (time.perf_counter() - t0) / steps * 1e3, result

    steps = max(3, min(args.steps, 10))
    e2e_steps = 3
    with ClockSampler(0) as clocks:
        prebuilt_ms, _ = timed(prebuilt_step, steps, args.warmup)
        batch_ms, batch_wall = timed(batch_step, steps, args.warmup)
        prebuilt_identical = all(torch.equal(a.view(torch.int32), b.view(torch.int32))
                                 for a, b in zip(d_plain, d_batch))
        for t in d_plain:
            t.fill_(0)
        percall_ms, _ = timed(percall_step, 3, 1)
        percall_identical = all(torch.equal(a.view(torch.int32), b.view(torch.int32))
                                for a, b in zip(d_plain, d_batch))
        host_ms, host_out = wall(lambda: batch.run_host(images), e2e_steps)
        public_ms, public_identical = None, None
        if public_loop:
            public_ms, public_out = wall(
                lambda: [public_call(nf, sp, im) for sp, im in zip(specs, images)], e2e_steps)
            public_identical = all(np.array_equal(a.view(np.uint32), b.view(np.uint32))
                                   for a, b in zip(public_out, host_out))
    launches = batch.launches
    batch.close()
    for plan in plans:
        plan.close()

    def rate(ms):
        return None if ms is None else round(pixels / (ms / 1e3) / 1e6, 3)

    return {
        "workload": "batch_mixed",
        "images": len(images),
        "pixels": pixels,
        "l2": "inputs total 3.7 GB (> 129 MB L2)",
        "unit": "Mpix/s",
        "batched": {"device": rate(batch_ms), "ms_per_step": round(batch_ms, 3),
                    "host_ms_per_step": round(batch_wall, 3),
                    "images_per_s": round(len(images) / (batch_ms / 1e3), 1),
                    "path": "ndf_batch_run: persistent family launches replayed from a CUDA graph",
                    "gpu_launches": launches},
        "plain_per_call": {"device": rate(percall_ms), "ms_per_step": round(percall_ms, 3),
                           "path": "per image: ndf_plan_create, ndf_plan_run on device buffers, "
                                   "ndf_plan_destroy"},
        "plain_prebuilt": {"device": rate(prebuilt_ms), "ms_per_step": round(prebuilt_ms, 3),
                           "path": "ndf_plan_run per image, plans built beforehand"},
        "speedup_vs_plain": {"device": round(percall_ms / batch_ms, 3),
                             "device_vs_prebuilt": round(prebuilt_ms / batch_ms, 3)},
        "e2e": {"batched": rate(host_ms), "ms_per_step": round(host_ms, 3),
                "path": "ndf_batch_run_host (pageable host arrays in and out)",
                "h2d_bytes_per_step": pixels * 4, "d2h_bytes_per_step": pixels * 4,
                "public_per_call": rate(public_ms),
                "public_ms_per_step": None if public_ms is None else round(public_ms, 3),
                "public_path": "public per-call API per image (nanmedian/nanpercentile/nanstd_filter)",
                "speedup_vs_public_per_call": None if public_ms is None else round(public_ms / host_ms, 3)},
        "outputs_identical": {"plain_per_call": bool(percall_identical),
                              "plain_prebuilt": bool(prebuilt_identical),
                              "public_per_call": public_identical},
        "autotune": {"keys": nf.autotune_entries(), "batch_create_s": round(batch_create_s, 3)},
        "clocks": clocks.summary(),
    }


def run_batch(args) -> None:
    import __graft_entry__

    __graft_entry__.build()
    r = batch_comparison(args)
    line = {
        "metric": METRIC,
        "value": r["batched"]["device"],
        "unit": "Mpix/s",
        "n_gpus": 1,
        "steps": max(3, min(args.steps, 10)),
        "warmup": args.warmup,
        "ms_per_step": r["batched"]["ms_per_step"],
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "f32",
        "data": "synthetic",
        "config": {"workload": "batch_mixed", "images": r["images"], "pixels": r["pixels"], "l2": r["l2"]},
        "e2e": {"value": r["e2e"]["batched"], "unit": "Mpix/s", "h2d_bytes_per_step": r["e2e"]["h2d_bytes_per_step"],
                "d2h_bytes_per_step": r["e2e"]["d2h_bytes_per_step"], "path": r["e2e"]["path"]},
        "batched": r,
        "clocks": r["clocks"],
        "gpu_launches": r["batched"]["gpu_launches"],
    }
    print(json.dumps(line))


# ---------------------------------------------------------------------------
# Precision study: nanstd against an exact (double-double) oracle.

def precision_study(rows: int = 192, width: int = 4096) -> dict:
    """Max relative error (and float32 ulp error) of nanstd on a strip of the
    1e4 + N(0, 1) image with 1% NaN, ddof=1, min_count=5, ignore_inf=True."""
    import ndfiltrs_gb300 as nf
    from oracle import oracle

    report = {"sample": f"{rows}x{width} strip of the seed-4 precision image (1e4 + N(0,1), 1% NaN)",
              "reference": "exact double-double window moments rounded once to float64"}
    for dtype in (np.float32, np.float64):
        image = np.ascontiguousarray(precision_image(width, dtype=dtype)[:rows])
        for size in ((31, 31), (7, 51)):
            opts = dict(omit_nan=True, ignore_inf=True, min_count=5)
            exact = oracle.exact_moments(image, "std", size, mode="reflect", ddof=1, **opts)
            finite = np.isfinite(exact) & (exact > 0)
            results = {}
            for name in ("fp32c", "fp64"):
                plan = nf.Plan(image.shape, dtype, "std", size, mode=["reflect"] * 2, parameter=1,
                               moments=name, **opts)
                results[f"gpu_{name}"] = plan.run_host(image)
                plan.close()
            results["cpu_reference_restatement"] = oracle.window_filter(
                image, "std", size, mode="reflect", parameter=1, **opts)
            entry = {}
            for name, value in results.items():
                nan_match = bool(np.array_equal(np.isnan(value), np.isnan(exact)))
                a = value[finite].astype(np.float64)
                e = exact[finite]
                rel = float(np.max(np.abs(a - e) / np.abs(e))) if a.size else 0.0
                item = {"max_rel_err": rel, "nan_pattern_matches": nan_match}
                if dtype == np.float32:
                    rounded = e.astype(np.float32)
                    ulp = np.spacing(np.abs(rounded)).astype(np.float64)
                    item["max_ulp_err"] = float(np.max(np.abs(a - rounded.astype(np.float64)) / ulp))
                entry[name] = item
            report[f"{np.dtype(dtype).name}_{size[0]}x{size[1]}"] = entry
    return report


# ---------------------------------------------------------------------------

def rotation_buffers(image_bytes: int) -> int:
    """Input buffers the device timing rotates over: together they exceed
    the 129 MB L2 three times over."""
    return max(4, -(-3 * 129 * 2**20 // image_bytes))


def workload_config(workload: str, spec, image: np.ndarray, world: int) -> dict:
    """The ``config`` object of a filter workload's line, identical in both
    arms (the reference arm's sample size is in its ``cpu_baseline``)."""
    n_buffers = rotation_buffers(image.nbytes)
    return {
        "workload": workload,
        "image": list(image.shape),
        "kind": spec.kind,
        "size": list(spec.window()),
        "footprint": None if spec.footprint_fn is None else int(spec.footprint().sum()),
        "origin": spec.origin,
        "percentile": spec.q if spec.kind == "percentile" else None,
        "mode": spec.mode,
        "omit_nan": spec.omit,
        "l2": f"device timing: inputs rotate over {n_buffers} device buffers "
              f"({n_buffers} x {image.nbytes / 1e6:.0f} MB > 129 MB L2)",
        "parallelism": f"replicas x{world}",
    }


def run_reference(args, spec, workload: str) -> None:
    image = spec.gen()
    steps, warmup = args.steps, args.warmup
    base = cpu_baseline(image, spec, budget_s=1.0)
    from oracle import oracle

    rows = base["rows"]
    strip = np.ascontiguousarray(image[:rows])
    threads = base["cores"]
    for _ in range(warmup):
        oracle_filter(oracle, spec, strip, threads)
    start = time.perf_counter()
    for _ in range(steps):
        oracle_filter(oracle, spec, strip, threads)
    elapsed = time.perf_counter() - start
    value = strip.size * steps / elapsed / 1e6
    base["value"] = round(value, 3)
    line = {
        "impl": "reference",
        "metric": METRIC,
        "value": round(value, 3),
        "unit": "Mpix/s",
        "n_gpus": args.gpus,
        "steps": steps,
        "warmup": warmup,
        "ms_per_step": round(elapsed / steps * 1e3, 3),
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "f32" if image.dtype == np.float32 else "f64",
        "data": "synthetic",
        "config": workload_config(workload, spec, image, args.gpus),
        "cpu_baseline": base,
        "e2e": {"value": round(value, 3), "unit": "Mpix/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))


MESH_WORKLOADS = {
    # SExtractor-rule mesh background of the 4096^2 sky image: 64 x 64 meshes,
    # 3 x 3 mesh median filter, natural-spline maps.
    "mesh_background_sextractor_64_4096_f32": dict(size=4096, box=64, options={}),
    # photutils rule set (3-sigma clip, SExtractor mode, IDW fill, truncated filter).
    "mesh_background_photutils_64_4096_f32": dict(
        size=4096, box=64, options=dict(estimator="sigma_clip", maxiters=10, statistic="mode", rms="std",
                                        min_valid_fraction=0.9, valid_count="retained", valid_base="box",
                                        fill="idw", filter_edge="truncate")),
}


def run_mesh(args) -> None:
    """Mesh background: device-resident pipeline timed with CUDA events
    (``ndf_mesh_background_device``: mesh statistics, host fill / filter, map
    interpolation), end to end through the public ``mesh_background``."""
    import ctypes

    import torch

    import __graft_entry__

    __graft_entry__.build()
    import ndfiltrs_gb300 as nf
    from ndfiltrs_gb300 import _core

    spec = MESH_WORKLOADS[args.workload]
    image = sky_image(spec["size"])
    box, options = spec["box"], dict(spec["options"])
    shape = image.shape
    pixels = image.size
    device = torch.device("cuda", 0)
    n_buffers = max(4, -(-3 * 129 * 2**20 // image.nbytes))
    buffers = [torch.from_numpy(np.roll(image, k * 97, axis=-1).copy()).to(device) for k in range(n_buffers)]
    out_bg, out_rms = torch.empty_like(buffers[0]), torch.empty_like(buffers[0])
    stream = torch.cuda.Stream(device)
    lib, _ = _core._load()
    estimator = options.get("estimator", "sextractor")
    rule = "sex" if estimator == "sextractor" else options.get("mode_estimator", "sex")
    config = _core.mesh_config(estimator, 3.0, 3.0, options.get("maxiters", 10), "median", "std",
                               options.get("statistic", "mode"), options.get("mode_estimator", "sex"),
                               2.5 if rule == "sex" else 3.0, options.get("rms", "std"),
                               options.get("min_valid_fraction", 0.5), options.get("valid_count", "finite"),
                               options.get("valid_base", "mesh"), options.get("fill", "nearest"), 10, 1.0,
                               options.get("filter_edge", "shrink"), None, "deviation", "spline")
    mesh_shape = tuple(-(-n // box) for n in shape)
    mb, mr = np.zeros(mesh_shape), np.zeros(mesh_shape)
    mv = np.zeros(mesh_shape, np.uint8)
    mf, mret = np.zeros(mesh_shape, np.int64), np.zeros(mesh_shape, np.int64)
    gl = np.zeros(2)
    u64 = lambda v: (ctypes.c_uint64 * len(v))(*v)
    ptr = lambda a, t: a.ctypes.data_as(ctypes.POINTER(t))

    def step(i: int) -> None:
        rc = lib.ndf_mesh_background_device(
            ctypes.c_void_p(buffers[i % n_buffers].data_ptr()), None, 0, 2, u64(list(shape)), u64([box, box]),
            u64([3, 3]), ctypes.byref(config), ctypes.c_void_p(out_bg.data_ptr()), ctypes.c_void_p(out_rms.data_ptr()),
            ptr(mb, ctypes.c_double), ptr(mr, ctypes.c_double), ptr(mv, ctypes.c_uint8), ptr(mf, ctypes.c_int64),
            ptr(mret, ctypes.c_int64), ptr(gl, ctypes.c_double), ctypes.c_void_p(stream.cuda_stream))
        if rc != 0:
            raise RuntimeError(lib.ndf_last_error().decode())

    for i in range(args.warmup):
        step(i)
    torch.cuda.synchronize()
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with ClockSampler(0) as clocks:
        start.record(stream)
        for i in range(args.steps):
            step(i)
        end.record(stream)
        torch.cuda.synchronize()
    elapsed_ms = start.elapsed_time(end)
    value = pixels * args.steps / (elapsed_ms / 1e3) / 1e6

    from oracle import oracle

    # Parity of the timed pipeline on the same image (maps and grids, bit for bit).
    got = nf.mesh_background(image, box, **options)
    want = oracle.mesh_background(image, box, 3, pearson=2.5 if rule == "sex" else 3.0, **options)
    check = all(np.array_equal(np.asarray(a).view(np.uint8), np.asarray(b).view(np.uint8))
                for a, b in zip(got[:7], want[:7]))
    e2e_steps = max(2, min(args.steps, 5))
    t0 = time.perf_counter()
    for _ in range(e2e_steps):
        nf.mesh_background(image, box, **options)
    e2e = pixels * e2e_steps / (time.perf_counter() - t0) / 1e6
    base = None
    if not args.no_cpu_baseline:
        threads = os.cpu_count() or 1
        runs = []
        for _ in range(3):
            t0 = time.perf_counter()
            oracle.mesh_background(image, box, 3, threads=threads, pearson=2.5 if rule == "sex" else 3.0, **options)
            runs.append(time.perf_counter() - t0)
        base = {"value": round(pixels / statistics.median(runs) / 1e6, 3), "unit": "Mpix/s", "cores": threads,
                "kind": "port",
                "sample": f"the whole {shape[0]}x{shape[1]} image, median of 3 calls, oracle restatement of "
                          f"MeshBackground::estimate + interpolate_into (meshes on {threads} threads)"}
    peak, peak_kind = measured_peak_hbm()
    achieved = 3 * image.itemsize * pixels / (elapsed_ms / args.steps / 1e3) / 1e9
    line = {
        "metric": "mesh background Mpix/s on 1 GB300",
        "value": round(value, 3),
        "unit": "Mpix/s",
        "n_gpus": 1,
        "steps": args.steps,
        "warmup": args.warmup,
        "ms_per_step": round(elapsed_ms / args.steps, 4),
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "f64",
        "data": "synthetic",
        "config": {"workload": args.workload, "image": list(shape), "box_size": box, "filter_size": 3,
                   "rules": options or "sextractor",
                   "l2": f"inputs rotate over {n_buffers} device buffers", "parallelism": "replicas x1"},
        "e2e": {"value": round(e2e, 3), "unit": "Mpix/s", "h2d_bytes_per_step": int(image.nbytes),
                "d2h_bytes_per_step": int(2 * image.nbytes), "path": "public mesh_background (ndf_mesh_background)",
                "steps": e2e_steps},
        "roofline": {"bound": "hbm", "achieved": round(achieved, 2), "peak": peak, "unit": "GB/s",
                     "frac": round(achieved / peak, 5), "traffic": None, "traffic_source": None,
                     "peak_source": peak_kind,
                     "note": "algorithmic bytes = 3 x 4 B/pixel (one read, two maps written); the per-mesh "
                             "statistics sort each mesh and sum in exact fixed point per block"},
        "cpu_baseline": base,
        "clocks": clocks.summary(),
        # Per call: the statistics and filter kernels, then per map (background,
        # rms) the spline's second-derivative and expansion passes along axis 0 and
        # the last axis's second derivatives, nodes and outputs.
        "gpu_launches": args.steps * 12,
        "parity_check_full": bool(check),
    }
    print(json.dumps(line))


def run_mesh_reference(args) -> None:
    """The oracle's mesh background on all host cores (the reference arm)."""
    from oracle import oracle

    spec = MESH_WORKLOADS[args.workload]
    image = sky_image(spec["size"])
    options = dict(spec["options"])
    rule = "sex" if options.get("estimator", "sextractor") == "sextractor" else options.get("mode_estimator", "sex")
    threads = os.cpu_count() or 1
    run = lambda: oracle.mesh_background(image, spec["box"], 3, threads=threads,
                                         pearson=2.5 if rule == "sex" else 3.0, **options)
    for _ in range(args.warmup):
        run()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        run()
    elapsed = time.perf_counter() - t0
    value = image.size * args.steps / elapsed / 1e6
    print(json.dumps({
        "impl": "reference", "metric": "mesh background Mpix/s on 1 GB300", "value": round(value, 3),
        "unit": "Mpix/s", "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": round(elapsed / args.steps * 1e3, 3), "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": args.workload, "image": list(image.shape)},
        "cpu_baseline": {"value": round(value, 3), "unit": "Mpix/s", "cores": threads, "kind": "port",
                         "sample": "the whole image per step"},
        "e2e": {"value": round(value, 3), "unit": "Mpix/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }))


def main() -> None:
    parser = argparse.ArgumentParser()
    parser.add_argument("--gpus", type=int, default=1)
    parser.add_argument("--steps", type=int, default=200)
    parser.add_argument("--warmup", type=int, default=5)
    parser.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    parser.add_argument("--workload", default=DEFAULT_WORKLOAD,
                        choices=sorted(WORKLOADS) + sorted(MESH_WORKLOADS) + ["batch_mixed"])
    parser.add_argument("--batch-images", type=int, default=512)
    parser.add_argument("--no-cpu-baseline", action="store_true")
    parser.add_argument("--precision", action=argparse.BooleanOptionalAction, default=True,
                        help="add the nanstd precision study to the line")
    parser.add_argument("--batch", action=argparse.BooleanOptionalAction, default=None,
                        help="add the mixed-size batch comparison (batched vs plain per-call GPU path) "
                             "to the line; on by default for the default workload")
    parser.add_argument("--pin-kernel", default=None,
                        help="kernel family the plan takes when it is a candidate (A/B comparisons)")
    args = parser.parse_args()
    args.warmup = max(3, args.warmup)
    if args.workload == "batch_mixed":
        run_batch(args)
        return
    if args.workload in MESH_WORKLOADS:
        if args.impl == "reference":
            run_mesh_reference(args)
        else:
            run_mesh(args)
        return
    spec = WORKLOADS[args.workload]

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))

    if args.impl == "reference":
        if rank == 0:
            run_reference(args, spec, args.workload)
        return

    import torch

    torch.cuda.set_device(local_rank)
    dist = None
    if world > 1:
        import torch.distributed as dist_module

        dist_module.init_process_group("nccl", device_id=torch.device("cuda", local_rank))
        dist = dist_module

    import __graft_entry__

    __graft_entry__.build()
    import ndfiltrs_gb300 as nf

    if args.pin_kernel:
        nf._core.pin_kernel(args.pin_kernel)
    image = spec.gen()  # every rank builds its own replica of the workload
    shape = image.shape
    pixels = image.size
    kind, mode = spec.kind, spec.mode

    def make_plan(shape_):
        return nf.Plan(shape_, image.dtype, kind, spec.window(), footprint=spec.footprint(),
                       origin=spec.origin, mode=[mode] * image.ndim, omit_nan=spec.omit,
                       ignore_inf=spec.ignore_inf, min_count=spec.min_count, parameter=spec.parameter,
                       percentile=spec.q, robust=spec.robust)

    plan = make_plan(shape)
    device = torch.device("cuda", local_rank)
    # Rotate over enough input buffers that together they exceed the 129 MB L2
    # three times over, so no step reads an input the previous ones left in L2.
    image_bytes = image.nbytes
    n_buffers = rotation_buffers(image_bytes)
    buffers = [torch.from_numpy(np.roll(image, k * 97, axis=-1).copy()).to(device) for k in range(n_buffers)]
    outputs = [torch.empty_like(buffers[0]) for _ in range(2)]
    stream = torch.cuda.Stream(device)
    handle = stream.cuda_stream

    def step(i: int) -> None:
        plan.run_device(buffers[i % n_buffers].data_ptr(), outputs[i % 2].data_ptr(), handle)

    for i in range(args.warmup):
        step(i)
    torch.cuda.synchronize()
    if dist is not None:
        dist.barrier()
    torch.cuda.synchronize()
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with ClockSampler(local_rank) as clocks:
        start.record(stream)
        for i in range(args.steps):
            step(i)
        end.record(stream)
        torch.cuda.synchronize()
    elapsed_ms = max_over_ranks(start.elapsed_time(end), dist, device)
    ms_per_step = elapsed_ms / args.steps
    value = replica_throughput(world, pixels, args.steps, elapsed_ms / 1e3)

    # Correctness spot check of the timed kernel against the oracle (not timed).
    check = None
    if rank == 0:
        from oracle import oracle

        rows = 64 if image.ndim < 3 else 4
        sample = np.ascontiguousarray(image[:rows])
        with make_plan(sample.shape) as sample_plan:
            gpu_sample = sample_plan.run_host(sample)
        expected = oracle_filter(oracle, spec, sample)
        ubits = np.uint32 if image.dtype == np.float32 else np.uint64
        check = bool(np.array_equal(gpu_sample.view(ubits), expected.view(ubits))) \
            if kind not in ("mean", "var", "std") else None  # FP32C moments: tolerance, not bits

    # End to end through the C-ABI host entry point with pinned buffers.
    host_in = torch.from_numpy(image).pin_memory()
    host_out = torch.empty(shape, dtype=torch.float32 if image.dtype == np.float32 else torch.float64).pin_memory()
    in_np, out_np = host_in.numpy(), host_out.numpy()
    e2e_steps = max(3, min(args.steps, 50))
    # Three untimed runs: the plan times its second (whole-array) and third
    # (row-band pipeline) host-buffer runs and keeps the faster form.
    for _ in range(3):
        plan.run_host_async(in_np, out_np, handle)
    if dist is not None:
        dist.barrier()
    t0 = time.perf_counter()
    for _ in range(e2e_steps):
        plan.run_host_async(in_np, out_np, handle)
    e2e_seconds = max_over_ranks(time.perf_counter() - t0, dist, device, barrier=False)
    e2e_value = replica_throughput(world, pixels, e2e_steps, e2e_seconds)

    # The drop-in boundary as the reference's Python layer calls it: one
    # `_core.window_filter` per image on pageable numpy arrays (the second
    # and later calls reuse the cached plan).
    core_call = None
    _core = nf._core
    if kind in _core.KINDS and kind not in _core.ROBUST_KINDS and kind != "percentile":
        def core_step():
            return _core.window_filter(image, kind, spec.window(), spec.footprint(), spec.origin,
                                       [mode] * image.ndim, 0.0, spec.omit, spec.ignore_inf, spec.min_count,
                                       spec.parameter)
        core_step()
        core_steps = max(3, min(args.steps, 10))
        t0 = time.perf_counter()
        for _ in range(core_steps):
            core_step()
        core_call = {"value": round(pixels * core_steps / (time.perf_counter() - t0) / 1e6, 3), "unit": "Mpix/s",
                     "path": "_core.window_filter per call (pageable numpy arrays in and out, cached plan)",
                     "steps": core_steps}

    peak, peak_kind = measured_peak_hbm()
    bytes_per_launch = pixels * image.itemsize * 2
    achieved = bytes_per_launch / (ms_per_step / 1e3) / 1e9
    base = None
    precision = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        base = cpu_baseline(image, spec)
    if rank == 0 and world == 1 and args.precision:
        precision = precision_study()
    batched = None
    if rank == 0 and world == 1 and (args.batch if args.batch is not None else args.workload == DEFAULT_WORKLOAD):
        batched = batch_comparison(args)

    if rank == 0:
        line = {
            "metric": METRIC,
            "value": round(value, 3),
            "unit": "Mpix/s",
            "n_gpus": world,
            "steps": args.steps,
            "warmup": args.warmup,
            "ms_per_step": round(ms_per_step, 4),
            "higher_is_better": True,
            "scaling": "weak",
            "vs_baseline": None,
            "dtype": "f32" if image.dtype == np.float32 else "f64",
            "data": "synthetic",
            "config": workload_config(args.workload, spec, image, world),
            "algorithm": plan.algorithm,
            "e2e": {
                "value": round(e2e_value, 3),
                "unit": "Mpix/s",
                "h2d_bytes_per_step": int(pixels * image.itemsize),
                "d2h_bytes_per_step": int(pixels * image.itemsize),
                "path": "ndf_plan_run_host (pinned host buffers, synchronized per step)",
                "steps": e2e_steps,
                "host_bands": plan.host_bands,
                "core_call": core_call,
            },
            "roofline": {
                "bound": "hbm",
                "achieved": round(achieved, 2),
                "peak": peak,
                "unit": "GB/s",
                "frac": round(achieved / peak, 5),
                "traffic": MEASURED_TRAFFIC.get(args.workload, (None,))[0],
                "traffic_source": MEASURED_TRAFFIC.get(args.workload, (None, None))[1],
                "peak_source": peak_kind,
                "note": f"selection is instruction-bound; algorithmic bytes = 2 x {image.itemsize} B/pixel "
                        "(one read, one write), halo re-reads excluded",
            },
            "issue_roofline": issue_roofline(args.workload, ms_per_step, int(torch.cuda.get_device_properties(
                device).multi_processor_count), clocks.summary().get("sm_mhz")),
            "cpu_baseline": base,
            "clocks": clocks.summary(),
            "gpu_launches": args.steps * LAUNCHES_PER_CALL.get(
                f"{plan.algorithm} {spec.kind}", LAUNCHES_PER_CALL.get(plan.algorithm, 1)),
            "nanstd_precision": precision,
            "batched": batched,
            "parity_check_rows64": check,
        }
        print(json.dumps(line))
    plan.close()
    if dist is not None:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
