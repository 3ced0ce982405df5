"""Autotuner for the decoders' launch shape.

Per codec it times every supported combination of
  warps_per_cta  chunks decoded by one CTA (one warp per chunk): 1, 2, 4, 8
  ring_slots     depth of the TMA input ring in 1 KiB slots: 4, 8
  cta_per_chunk  RLE: a whole CTA per chunk instead of one warp, whatever their number
on a resident sample of the caller's chunks, installs with codag_set_tune the fastest if it is faster
than the library's own shape by more than such times differ from one another (else that one), and caches it in
a JSON file keyed by GPU name and codec, so later runs on the same kind of GPU skip the search.
Deflate chunks and batched plans have one shape, which the tune fields do not change; nor do they
change anything for RLE chunks that have a CTA each without being asked (include/codag.h), where
all candidates are the same kernel and only the difference of the times would choose.
"""
from __future__ import annotations

import itertools
import json
import os
from pathlib import Path

import torch

from . import native

CACHE = Path(os.environ.get("CODAG_TUNE_CACHE", Path(__file__).resolve().parent / "tune_cache.json"))


# what the library starts with, and by how much another shape has to be faster: medians of three calls of one kernel
# differ by up to 3%
DEFAULT = {native.RLEV1: (8, 4, 10, 0), native.RLEV2: (8, 4, 10, 0), native.DEFLATE: (2, 2, 9, 0)}
MARGIN = 0.95


def candidates(codec: int):
    if codec == native.DEFLATE:
        return [DEFAULT[codec]]
    # one warp per chunk, or one CTA per chunk
    return list(itertools.product((1, 2, 4, 8), (4, 8), (10,), (0,))) + [(8, 4, 10, 1)]


def batch_candidates():
    """Launch shapes of the batched kernel (warps_per_cta, ring_slots, lut_bits, cta_per_chunk,
    table_global): there is one, which a plan picks by the sizes of its files."""
    return [(8, 4, 10, 0, 0)]


def _key(codec: int, tag: str) -> str:
    return f"{torch.cuda.get_device_name()}|codec{codec}|{tag}|margin"


def load_cached(codec: int, tag: str = "plain"):
    try:
        return json.loads(CACHE.read_text()).get(_key(codec, tag))
    except (OSError, ValueError):
        return None


def store_cached(codec: int, tag: str, shape) -> None:
    try:
        data = json.loads(CACHE.read_text())
    except (OSError, ValueError):
        data = {}
    data[_key(codec, tag)] = list(shape)
    # written whole and renamed into place: ranks of one job may store at the same time
    tmp = CACHE.with_name(f"{CACHE.name}.{os.getpid()}.tmp")
    try:
        tmp.write_text(json.dumps(data, indent=1, sort_keys=True))
        os.replace(tmp, CACHE)
    except OSError:
        pass


def time_call(fn, reps: int = 3) -> float:
    """Median device time (s) of fn() on the current stream after one warm-up call."""
    fn()
    torch.cuda.synchronize()
    ts = []
    for _ in range(reps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        fn()
        b.record()
        torch.cuda.synchronize()
        ts.append(a.elapsed_time(b) / 1e3)
    ts.sort()
    return ts[len(ts) // 2]


def autotune(codec: int, run, tag: str = "plain", use_cache: bool = True, verbose: bool = False):
    """Search the launch shape of `codec` with `run()` (one decode of a resident sample),
    install the winner and return (shape, {shape: seconds}); without a clear winner the default."""
    if use_cache:
        hit = load_cached(codec, tag)
        if hit:
            native.set_tune(codec, *hit)
            return tuple(hit), {}
    results = {}
    for shape in candidates(codec):
        native.set_tune(codec, *shape)
        results[shape] = time_call(run)
        if verbose:
            print(f"codec {codec} shape {shape}: {results[shape] * 1e3:.3f} ms", flush=True)
    best = min(results, key=results.get)
    if results[best] > MARGIN * results[DEFAULT[codec]]:
        best = DEFAULT[codec]
    native.set_tune(codec, *best)
    store_cached(codec, tag, best)
    return best, results
