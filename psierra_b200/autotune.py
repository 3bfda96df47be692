"""Launch-shape autotuner of the persistent assembly kernel.

Three knobs change the speed of ``psx_tet4_assemble`` / ``psx_tet10_assemble`` on a given
mesh without changing a single output bit (each K and f entry is summed by one owner in
a fixed order whatever the schedule): the lag of the task queue in use (granules between
an element tile and the gathers it completes: too small and gathers wait for elements
still in flight, too large and the ring outgrows L2), the ring slack (room for element
tiles in flight before they must wait for old gathers), the number of persistent
blocks per SM and, for Tet4 FP32 tangent sweeps, whether element tiles and gathers run
in separate warps (the warp-specialised kernel, whose ring is sized by the same lag and
slack) or in the same ones.  ``tune`` times each candidate with CUDA events on the
caller's stream and keeps the fastest; results are cached per device, element type,
mesh size and precision, in memory and optionally in a JSON file.

Sweeps that also run in two launches without a queue are timed that way last, and keep it when
it is faster.  That changes no bit either, but for the FP32 tangents of meshes large enough for
point records (``MeshPattern.POINT_ELEMENTS_FP32``), whose sums are associated differently.
"""
from __future__ import annotations

import json
import os

import torch

from psierra_b200.assembler import raise_if_wait_gave_up

DEFAULT_LAGS = (8, 12, 16, 24)
DEFAULT_BLOCKS = (2,)
DEFAULT_SLACKS = (6, 12, 20)

DEFAULT_SPLITS = (True, False)

_cache: dict[str, tuple] = {}


# What was compared.  An entry of an earlier set does not say which of today's ways is the fastest
# (before the two launches every entry named a queue), so it is not used: the mesh is timed again.
_WAYS = "queue,two-pass"


def _key(asm, precision: str, want_f: bool, want_k: bool) -> str:
    name = torch.cuda.get_device_name(asm.device)
    return f"{name}|npe{asm.npe}|E{asm.n_elements}|N{asm.n_nodes}|{precision}|f{int(want_f)}k{int(want_k)}|{_WAYS}"


def _time(asm, u, precision, want_f, want_k, f, k, reps: int) -> float:
    for _ in range(2):
        asm.assemble(u, want_f=want_f, want_k=want_k, precision=precision, f_out=f, k_out=k, check_status=False)
    a = torch.cuda.Event(enable_timing=True)
    b = torch.cuda.Event(enable_timing=True)
    a.record()
    for _ in range(reps):
        asm.assemble(u, want_f=want_f, want_k=want_k, precision=precision, f_out=f, k_out=k, check_status=False)
    b.record()
    b.synchronize()
    # the status of the last timed call: a candidate whose bounded wait gave up is not a
    # valid launch shape
    raise_if_wait_gave_up(asm.status_counts()[3])
    return a.elapsed_time(b) / reps


def _apply(asm, want_k: bool, lag: int, bps: int, slack: int, split: bool | None = None) -> None:
    """Queue the sweeps tuned, in this shape; the others stay queued or in two passes as they are."""
    other_queued = getattr(asm.pattern, "queued_f" if want_k else "queued_k", True)
    if want_k:
        asm.set_queue(lag=lag, blocks_per_sm=bps, ring_slack=slack, split=split)
    else:
        asm.set_queue(lag_f=lag, blocks_per_sm=bps, ring_slack=slack)
    if not other_queued:  # the blocks per SM queue them too
        asm.set_two_pass(f=want_k, k=not want_k)


def _result(entry: tuple, ms: float | None, table: dict) -> dict:
    return dict(zip(("lag", "blocks_per_sm", "ring_slack", "split", "two_pass"), entry), ms=ms, table=table)


def tune(asm, u: torch.Tensor, precision: str | None = None, want_f: bool = True, want_k: bool = True,
         lags=DEFAULT_LAGS, blocks=DEFAULT_BLOCKS, slacks=DEFAULT_SLACKS, splits=DEFAULT_SPLITS, reps: int = 5,
         cache_file: str | None = None) -> dict:
    """Pick the queue's (lag, blocks_per_sm, ring_slack, split) or two passes for ``asm`` by timing;
    applies and returns the choice.

    The lag tuned is that of the queue the sweep uses (the K queue when ``want_k``, else
    the f queue).  ``splits`` is swept only for Tet4 FP32 tangent sweeps (the only ones
    with a warp-specialised kernel); elsewhere split is left as it is.  Returns
    ``{"two_pass", "ms", "lag", "blocks_per_sm", "ring_slack", "split", "table": {(lag, bps, slack,
    split): ms}}``: whether two passes won, the time of what runs now, the best queue and the
    queues' times.  With a cached entry for the same key nothing is timed (``ms`` is None).

    A tangent's queue holds for both precisions of the pattern, as its lag does.
    """
    prec = precision or asm.precision
    key = _key(asm, prec, want_f, want_k)
    disk = {}
    if cache_file and os.path.exists(cache_file):
        with open(cache_file) as fh:
            disk = json.load(fh)
    hit = _cache.get(key) or (tuple(disk[key]) if key in disk else None)
    if hit is not None:
        _apply(asm, want_k, *hit[:4])
        if hit[4]:
            asm.set_two_pass(f=not want_k, k=want_k)
        return _result(hit, None, {})
    f = asm.new_f() if want_f else None
    k = asm.new_k(prec) if want_k else None
    has_split = asm.npe == 4 and want_k and prec == "fp32-mixed"
    split_opts = tuple(bool(x) for x in splits) if has_split else (asm.pattern.split,)
    table = {}
    for split in split_opts:
        for lag in lags:
            for bps in blocks:
                for slack in slacks:
                    _apply(asm, want_k, lag, bps, slack, split)
                    table[(lag, bps, slack, split)] = _time(asm, u, prec, want_f, want_k, f, k, reps)
    best = min(table, key=table.get)
    two_pass, ms = False, table[best]
    _apply(asm, want_k, *best)
    if hasattr(asm, "set_two_pass"):
        # sweeps that also run in two passes, without a queue: keep the faster way
        asm.set_two_pass(f=not want_k, k=want_k)
        if asm.pattern.tangent_in_two_passes(prec) if want_k else asm.pattern.two_pass:
            passes_ms = _time(asm, u, prec, want_f, want_k, f, k, reps)
            two_pass, ms = passes_ms < ms, min(passes_ms, ms)
        if not two_pass:
            _apply(asm, want_k, *best)
    entry = best + (two_pass,)
    _cache[key] = entry
    if cache_file:
        disk[key] = list(entry)
        with open(cache_file, "w") as fh:
            json.dump(disk, fh, indent=1, sort_keys=True)
    return _result(entry, ms, table)
