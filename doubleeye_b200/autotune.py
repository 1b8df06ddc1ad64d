"""Autotuner for the dense pipeline's launch shapes.

The kernels leave the arithmetic fixed; these knobs only change how work is laid
onto the GPU, so every setting gives bit-identical results:

  rows_ctas_per_sm  resident row-kernel CTAs per SM (persistent grid size)
  cols_kt           streaming column kernel: disparities per lane (0 = by batch size)
  cols_pf           streaming column kernel: image rows loaded ahead of use
  cols_cta          streaming column kernel: threads per CTA (0 = by batch size)
  solve_threads     row solve: two pixels a thread (512), four (256), 0 = by row width
  batch_streams     parts a batch runs as on concurrent streams
  cols_async        streaming column kernel: prefetch through shared memory (1) or
                    registers (0)

A single pair of usual size takes a column kernel of another form while the four cols_*
knobs are at their defaults; any other setting of one of them means the streaming kernel.

``tune`` times a batch under a coordinate-descent search over these values (CUDA
events, warm-up first) and returns the fastest setting; ``Tuner`` caches the choice
per device and workload signature (pair shapes, disparity ranges, iterations) in a
JSON file next to the library, so a workload is tuned once per machine.
"""
from __future__ import annotations

import json
import os
import threading

from . import _lib

KNOBS = {
    "rows_ctas_per_sm": [4, 8, 32],
    "cols_kt": [0, 4, 8, 16],
    "cols_pf": [0, 4, 8, 16],
    "cols_cta": [0, 128, 256],
    "solve_threads": [0, 256, 512],          # (128 is the same launch as 256)
    "batch_streams": [1, 2, 3, 4],
    "cols_async": [1, 0],
}
CACHE = os.path.join(_lib.PKG, "_lib", "autotune.json")


def current() -> dict:
    return {k: _lib.get_param(k) for k in KNOBS}


def apply(knobs: dict) -> None:
    for k, v in knobs.items():
        _lib.set_param(k, int(v))


def signature(cfg, shapes) -> str:
    """Workload key: sorted (W, H, D) multiset plus the iteration count."""
    from collections import Counter
    D0 = cfg.dmax - cfg.dmin + 1
    norm = Counter((int(W), int(H), int(d) - cfg.dmin + 1 if d else D0) for W, H, d in shapes)
    body = ",".join(f"{W}x{H}xD{D}*{n}" for (W, H, D), n in sorted(norm.items()))
    return f"iters{cfg.iters}:lrc{cfg.lrc}:{body}"


def _time(run, reps: int, warmup: int) -> float:
    import torch
    for _ in range(warmup):
        run()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(reps):
        run()
    e1.record()
    torch.cuda.synchronize()
    return e0.elapsed_time(e1) / reps


def tune(run, reps: int = 3, warmup: int = 2, rounds: int = 2) -> tuple[dict, float]:
    """Coordinate descent from the current setting: for each knob in turn keep the
    fastest value, two rounds.  ``run`` enqueues one batch.  A winner that differs
    from the starting setting is then timed against it in alternation (the clock and
    the memory system drift by a percent or two within a run, so one short timing
    per trial can pick a setting that is not faster) and kept only if it is at least
    1% faster there.  Leaves the chosen setting applied and returns it with its time
    (ms per batch)."""
    start = current()
    best = dict(start)
    apply(best)
    best_ms = _time(run, reps, warmup)
    for _ in range(rounds):
        improved = False
        for k, values in KNOBS.items():
            for v in values:
                if v == best[k]:
                    continue
                trial = dict(best, **{k: v})
                apply(trial)
                ms = _time(run, reps, warmup)
                if ms < best_ms * 0.99:
                    best, best_ms, improved = trial, ms, True
            apply(best)
        if not improved:
            break
    if best != start:
        t_start = t_best = 0.0
        for _ in range(2):
            apply(start)
            t_start += _time(run, reps, 1)
            apply(best)
            t_best += _time(run, reps, 1)
        if t_best > 0.99 * t_start:
            best, best_ms = start, t_start / 2
        else:
            best_ms = t_best / 2
    apply(best)
    return best, best_ms


class Tuner:
    """Per-device, per-workload knob cache (JSON next to the library)."""

    _lock = threading.Lock()

    def __init__(self, path: str = CACHE):
        self.path = path
        self.table = {}
        if os.path.exists(path):
            try:
                with open(path) as f:
                    self.table = json.load(f)
            except (OSError, ValueError):
                self.table = {}

    @staticmethod
    def _device_key() -> str:
        import torch
        p = torch.cuda.get_device_properties(torch.cuda.current_device())
        return f"{p.name}:{p.multi_processor_count}"

    def lookup(self, sig: str):
        return self.table.get(self._device_key(), {}).get(sig)

    def record(self, sig: str, knobs: dict, ms: float) -> None:
        with self._lock:
            self.table.setdefault(self._device_key(), {})[sig] = dict(knobs, ms=ms)
            try:
                tmp = self.path + ".tmp"
                with open(tmp, "w") as f:
                    json.dump(self.table, f, indent=1, sort_keys=True)
                os.replace(tmp, self.path)
            except OSError:
                pass

    def ensure(self, sig: str, run) -> dict:
        """The cached setting for ``sig`` (applied), tuning it first if absent."""
        hit = self.lookup(sig)
        if hit is None or any(k not in hit for k in KNOBS):    # absent, or older knob set
            knobs, ms = tune(run)
            self.record(sig, knobs, ms)
            return knobs
        knobs = {k: hit[k] for k in KNOBS}
        apply(knobs)
        return knobs
