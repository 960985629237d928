"""Autotuner for the compositing kernels' launch shape.

Times the library's own choice (the launch rule of csrc/render.cu) and then sweeps
pixels per thread {1, 2, 4} x records per shared-memory batch {64, 128, 256} for the
forward and the backward render kernels on a caller's own step (one forward +
backward on representative views), timing each with the library's per-stage CUDA
events; then, with the fastest forward shape, the forward's long-tile threshold among
the caller's candidates (fgs_set_render_split).  The fastest forward and the fastest
backward are installed for the process, the library's choice where nothing beats it.
(The backward's kernels do not depend on the batch: its times at one pixel count
differ by noise only, and cost nothing beside the forward's.)  Results are cached per
workload key.
"""
import torch

from . import _lib

PPT = (1, 2, 4)
BATCH = (64, 128, 256)
_cache = {}


def tune_render(run_step, key=None, steps=3, warmup=1, splits=((0, 0),)):
    """run_step() performs one forward + backward through this library.

    splits: candidate (min_records, band_shape) long-tile settings of the forward
    (fgs_set_render_split), tried with the best forward shape; the fastest is installed
    (table keys ("split", min_records, band_shape); ("split", "library") is the library's
    choice of shape and long tiles).
    Returns ((fwd_ppt, fwd_batch, bwd_ppt, bwd_batch), {(ppt, batch): (fwd_ms, bwd_ms)})."""
    if key is not None and key in _cache:
        best, table, split = _cache[key]
        _lib.set_render_config(*best)
        _lib.set_render_split(*split)
        return best, table
    _lib.set_render_config()
    _lib.set_render_split()
    rule, rule_split = _lib.get_render_config(), _lib.get_render_split()
    table = {("split", "library"): _time(run_step, steps, warmup)}
    rule_fwd, rule_bwd = table[("split", "library")]
    shapes = {}
    _lib.set_render_split(*splits[0])
    for p in PPT:
        for b in BATCH:
            _lib.set_render_config(p, b, p, b)
            shapes[(p, b)] = _time(run_step, steps, warmup)
    table.update(shapes)
    bf = min(shapes, key=lambda c: shapes[c][0])
    bb = min(shapes, key=lambda c: shapes[c][1])
    _lib.set_render_config(*bf, *bb)
    split, fwd = None, None
    for sp in splits:
        _lib.set_render_split(*sp)
        ms = _time(run_step, steps, warmup)[0]
        table[("split",) + tuple(sp)] = (ms, 0.0)
        if fwd is None or ms < fwd:
            split, fwd = sp, ms
    if rule_fwd <= fwd:
        bf, split = rule[:2], rule_split
    if rule_bwd <= shapes[bb][1]:
        bb = rule[2:]
    best = tuple(bf) + tuple(bb)
    _lib.set_render_config(*best)
    _lib.set_render_split(*split)
    if key is not None:
        _cache[key] = (best, table, split)
    return best, table


def _time(run_step, steps, warmup):
    """(forward, backward) compositing milliseconds per step."""
    for _ in range(warmup):
        run_step()
    torch.cuda.synchronize()
    _lib.profile_read(reset=True)
    _lib.profile_enable(True)
    for _ in range(steps):
        run_step()
    torch.cuda.synchronize()
    _lib.profile_enable(False)
    prof = _lib.profile_read(reset=True)
    return prof["render_fwd"][0] / steps, prof["render_bwd"][0] / steps
