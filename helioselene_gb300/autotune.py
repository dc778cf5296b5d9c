"""Window and accumulation autotuner for the batched and per-call MSM paths.

For every size class (powers of two from 2^6 to 2^20) it times, on the GPU, a
batch of MSMs of that size over candidate window widths c (a hill-climb that
starts from the previous class's best); then, at the best c, the bucket
accumulation form: 0, 1 or 2 batch-affine rounds (the wave of pairwise
additions that share one inversion, hs_context_set_batch_affine).  The library's
defaults, which depend on how many MSMs run together, are timed beside them: a
class gets a rule only where the rule beats them in the batch by MIN_GAIN and
does not slow one MSM of that size by itself, since a rule holds for both.
The table becomes the context's rules (hs_context_set_rule: c per class, and
the rounds of plans whose entries lie mostly in that class) and can be saved
to / loaded from a JSON cache keyed by device name and library build.

The reference hard-codes its window by n (helios/src/x64/helios_msm_vartime.cpp:248-263)
and its autotune times only backends at n = 16 (src/dispatch.cpp:381-421); here
the choice is measured per size class on the device that will run it.
"""

from __future__ import annotations

import hashlib
import json
import time
from pathlib import Path
from typing import Callable, Dict, Iterable, Optional

import numpy as np

from . import _lib as L

DEFAULT_CANDIDATES = tuple(range(4, 17))
ROUND_CANDIDATES = (0, 1, 2)
MIN_GAIN = 0.03   # of the defaults' time in the batch
LONE_LOSS = 0.01  # of the defaults' time of one MSM: what the timing does not resolve


def _classes(n_min: int, n_max: int):
    k = max(1, int(np.floor(np.log2(max(1, n_min)))))
    while (1 << k) <= n_max:
        lo, hi = 1 << k, (1 << (k + 1)) - 1
        yield lo, hi
        k += 1


def _climb(measure: Callable[[int], float], cands: list, start: int) -> int:
    """the best width, walked outward from start until two neighbours in a row are slower"""
    best = start
    for direction in (+1, -1):
        worse = 0
        c = start + direction
        while cands[0] <= c <= cands[-1] and worse < 2:
            if measure(c) < measure(best):
                best, worse = c, 0
            else:
                worse += 1
            c += direction
    return best


def _rule(batch: Callable, lone: Callable, cands: list, start: int):
    """(best width of the batch, the class's rule or None) from the timings batch(form) and
    lone(form), where a form is (c, rounds), or None for the library's defaults"""
    best_c = _climb(lambda c: batch((c, 0)), cands, start)
    form = min(((best_c, r) for r in ROUND_CANDIDATES), key=batch)
    if batch(form) > (1 - MIN_GAIN) * batch(None) or lone(form) > (1 + LONE_LOSS) * lone(None):
        return best_c, None
    return best_c, {"c": form[0], "rounds": form[1]}


def tune(ctx, curve: int, n_min: int = 64, n_max: int = 1 << 20, candidates: Iterable[int] = DEFAULT_CANDIDATES,
         points_per_class: int = 1 << 20, reps: int = 3, seed: int = 1) -> Dict[str, dict]:
    """Return {"lo-hi": {"c": c, "rounds": r}} for each size class in which a rule beats the
    library's defaults, measured with batched device MSMs and with single ones."""
    import torch

    from .workload import ORDER, random_field_bytes, random_scalars
    rng = np.random.default_rng(seed)
    table = {}
    cands = sorted(set(candidates))
    start = min(cands, key=lambda c: abs(c - 8))
    stream = torch.cuda.ExternalStream(ctx.stream)
    for lo, hi in _classes(n_min, n_max):
        n = lo + (hi - lo) // 2
        count = max(1, min(256, points_per_class // n))
        total = n * count
        d_u = torch.from_numpy(random_field_bytes(rng, total).reshape(-1)).cuda()
        d_pts = torch.empty(total * 64, dtype=torch.uint8, device="cuda")
        d_sc = torch.from_numpy(random_scalars(rng, total, ORDER[curve]).reshape(-1)).cuda()
        d_out = torch.empty(count * 120, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        ctx.map_to_curve_device(curve, d_u.data_ptr(), total, d_pts.data_ptr())
        timed = {}

        def measure(form, sizes):
            key = (form, len(sizes))
            if key not in timed:
                ctx.set_window(curve, 0, 0, 0)
                if form is not None:
                    ctx.set_window(curve, 1, 1 << 31, *form)

                def run():
                    if len(sizes) == 1:
                        ctx.msm_device(curve, d_sc.data_ptr(), d_pts.data_ptr(), n, d_out.data_ptr())
                    else:
                        ctx.msm_batch_device(curve, sizes, d_sc.data_ptr(), d_pts.data_ptr(), d_out.data_ptr())

                run()
                stream.synchronize()
                ts = []
                for _ in range(reps):
                    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                    a.record(stream)
                    run()
                    b.record(stream)
                    stream.synchronize()
                    ts.append(a.elapsed_time(b))
                timed[key] = min(ts)
            return timed[key]

        start, rule = _rule(lambda f: measure(f, [n] * count), lambda f: measure(f, [n]), cands, start)
        if rule:
            table[f"{lo}-{hi}"] = rule
        del d_u, d_pts, d_sc, d_out
    ctx.set_window(curve, 0, 0, 0)
    return table


def apply(ctx, curve: int, table: Dict[str, object]) -> None:
    """install a table: entries {"c", "rounds"} (or a bare window width)"""
    ctx.set_window(curve, 0, 0, 0)
    for key, v in table.items():
        lo, hi = (int(x) for x in key.split("-"))
        if isinstance(v, dict):
            ctx.set_window(curve, lo, hi, int(v["c"]), int(v.get("rounds", -1)))
        else:
            ctx.set_window(curve, lo, hi, int(v))


def _library_id() -> str:
    """the build whose kernels and defaults a table was measured with"""
    return hashlib.sha256(Path(L.LIB_PATH).read_bytes()).hexdigest()[:16]


def load_or_tune(ctx, cache: Optional[Path] = None, n_max: int = 1 << 20, **kw) -> dict:
    """Tables for both curves from the cache (matching device and library) or freshly tuned."""
    import torch
    dev = torch.cuda.get_device_name(ctx.device)
    library = _library_id()
    data = {}
    if cache and Path(cache).exists():
        try:
            data = json.loads(Path(cache).read_text())
        except (OSError, ValueError):
            data = {}
    entry = data.get(dev)
    if not entry or entry.get("library") != library or entry.get("n_max", 0) < n_max:
        t0 = time.time()
        entry = {"n_max": n_max, "library": library, "helios": tune(ctx, L.HELIOS, n_max=n_max, **kw),
                 "selene": tune(ctx, L.SELENE, n_max=n_max, **kw), "seconds": round(time.time() - t0, 2)}
        data[dev] = entry
        if cache:
            try:
                Path(cache).write_text(json.dumps(data, indent=1, sort_keys=True) + "\n")
            except OSError:
                pass
    apply(ctx, L.HELIOS, entry["helios"])
    apply(ctx, L.SELENE, entry["selene"])
    return entry
