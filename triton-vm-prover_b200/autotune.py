"""Autotuner for the table-commitment kernels.

Times candidate values of the library's tuning knobs (tvmc_set_tuning) on the
caller's own table shapes, keeps the fastest, and persists the choice in a JSON
cache keyed by device name, build of the library and shape, so later processes
start tuned (a choice made among another build's kernels is not taken over):

    lde_mid_variant     fused LDE middle kernel: per-coset global twiddles (1) or
                        inter-pass twiddles shared across cosets in shared memory (2),
                        or 2^8- and 2^10-point passes on the tensor cores (0)
    lde_mid_ctas        its resident CTAs/SM (2, 3)
    lde_split_l1        the LDE's four-step split N = n1 * n2 (the default, balanced,
                        n1 = N^(1/2) / 4, or n1 = 2^12 where valid)
    ntt_tile_log        words an NTT pass CTA moves per tile (2^12 .. 2^14)
    batch_streams       worker streams of a tvmc_batch (1 .. 16)
    batch_multi_hash    one multi-table row-hash launch for a batch (1) or per-table hashes (2)
    frugal_stripe_cols  columns per frugal stripe (multiples of 10)

Every candidate computes the same bits (the knobs only change scheduling and
register allocation), so tuning never affects results.
"""
from __future__ import annotations

import functools
import hashlib
import json
import os
import time

import tvmc

CACHE = os.environ.get("TVMC_TUNING_CACHE", os.path.join(os.path.expanduser("~"), ".cache", "tvmc",
                                                          "tuning.json"))


def _device_name() -> str:
    try:
        import torch
        return torch.cuda.get_device_name()
    except Exception:
        return "cuda"


@functools.lru_cache(maxsize=None)
def _build() -> str:
    with open(tvmc.LIB_PATH, "rb") as f:
        return hashlib.sha256(f.read()).hexdigest()[:16]


def _key(kind: str, shape: str) -> str:
    return f"{_device_name()}|{_build()}|{kind}|{shape}"


def load(path: str = CACHE) -> dict:
    try:
        with open(path) as f:
            return json.load(f)
    except (OSError, ValueError):
        return {}


def save(db: dict, path: str = CACHE) -> None:
    os.makedirs(os.path.dirname(path), exist_ok=True)
    tmp = path + ".tmp"
    with open(tmp, "w") as f:
        json.dump(db, f, indent=1, sort_keys=True)
    os.replace(tmp, path)


def apply(knobs: dict) -> None:
    for k, v in knobs.items():
        tvmc.set_tuning(k, int(v))


def _time(fn, reps: int = 3) -> float:
    import torch
    fn()  # warm-up (also builds twiddle tables)
    torch.cuda.synchronize()
    best = float("inf")
    for _ in range(reps):
        t0 = time.perf_counter()
        fn()
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t0)
    return best


def lde_candidates(log_n: int):
    """The LDE knob combinations worth timing for a trace of 2^log_n rows."""
    balanced = (log_n + 1) // 2
    splits = [l1 for l1 in dict.fromkeys((balanced, log_n // 2 - 2, 12)) if 6 <= l1 <= 12 and 6 <= log_n - l1 <= 12]

    def combine(variants, ctas, splits):
        return [{"lde_mid_variant": v, "lde_mid_ctas": c, "lde_split_l1": s, "ntt_tile_log": t}
                for v in variants for c in ctas for s in splits for t in (12, 13, 14)]

    # On the tensor cores (variant 0) the default split is the library's own choice,
    # so the balanced one is a candidate beside it; K2 takes one CTA per SM there.
    # The register networks' default split is the balanced one.
    return combine((0,), (3,), [0] + splits) + combine((1, 2), (2, 3), [0] + [s for s in splits if s != balanced])


def tune_commit(trace_ptr: int, trace_len: int, width: int, expansion: int = 4, offset: int = 7,
                stream=None, path: str = CACHE, force: bool = False) -> dict:
    """Tune the plain commit of one device-resident column-major table: the LDE
    knobs, on the LDE alone (up to 64 of its columns)."""
    import torch
    key = _key("commit", f"{trace_len}x{width}x{expansion}")
    db = load(path)
    if key in db and not force:
        apply(db[key]["knobs"])
        return db[key]
    log_n = trace_len.bit_length() - 1
    cols = max(1, min(width, 64))
    out = torch.empty(cols * trace_len * expansion, dtype=torch.int64, device="cuda")
    lde_s = {}
    for knobs in lde_candidates(log_n):
        apply(knobs)
        lde_s[tuple(knobs.values())] = _time(
            lambda: tvmc.lde_gpu(trace_ptr, cols, trace_len, out.data_ptr(), trace_len * expansion, offset,
                                 stream=stream))
    del out
    best_lde = dict(zip(("lde_mid_variant", "lde_mid_ctas", "lde_split_l1", "ntt_tile_log"),
                        min(lde_s, key=lde_s.get)))
    entry = {"knobs": best_lde, "seconds": {"lde": {",".join(map(str, k)): v for k, v in lde_s.items()}}}
    apply(entry["knobs"])
    db[key] = entry
    save(db, path)
    return entry


def tune_batch(shapes, fill, path: str = CACHE, force: bool = False, candidates=(1, 2, 4, 8, 16)) -> dict:
    """Tune batch_streams for a tvmc.Batch of `shapes`; fill(batch) loads inputs."""
    key = _key("batch", ",".join(f"{s[0]}x{s[1]}" for s in shapes))
    db = load(path)
    if key in db and not force:
        apply(db[key]["knobs"])
        return db[key]
    results = {}
    for multi in (1, 2):
        for k in candidates:
            tvmc.set_tuning("batch_streams", k)
            tvmc.set_tuning("batch_multi_hash", multi)
            with tvmc.Batch(shapes) as b:
                fill(b)
                results[(multi, k)] = _time(b.run)
    best = min(results, key=results.get)
    entry = {"knobs": {"batch_multi_hash": best[0], "batch_streams": best[1]},
             "seconds": {f"{m},{k}": v for (m, k), v in results.items()}}
    apply(entry["knobs"])
    db[key] = entry
    save(db, path)
    return entry


def tune_frugal(trace_ptr: int, trace_len: int, width: int, expansion: int = 4, offset: int = 7,
                path: str = CACHE, force: bool = False, candidates=(10, 20, 40, 80)) -> dict:
    key = _key("frugal", f"{trace_len}x{width}x{expansion}")
    db = load(path)
    if key in db and not force:
        apply(db[key]["knobs"])
        return db[key]
    results = {}
    for sc in candidates:
        tvmc.set_tuning("frugal_stripe_cols", sc)

        def run():
            with tvmc.Commitment(trace_ptr, width=width, trace_len=trace_len, device_ptr=True,
                                 expansion=expansion, offset=offset, frugal=True) as c:
                c.sync()

        results[sc] = _time(run, reps=2)
    best = min(results, key=results.get)
    entry = {"knobs": {"frugal_stripe_cols": best}, "seconds": {str(k): v for k, v in results.items()}}
    apply(entry["knobs"])
    db[key] = entry
    save(db, path)
    return entry
