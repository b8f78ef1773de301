"""Pick the fused kernel's shape per (model, stencil, grid size) by timing.

The fused float32 form has several kernels -- the TMA pipeline (64 x 32
regions, one persistent CTA per SM, with 4 x 1 or 2 x 2 nodes per thread)
and the cp.async kernels (64 x 32 regions with two CTAs per SM, or 64 x 64
regions) -- and a temporal-block depth K (time steps per launch: 2, 3, 4
or 8).  Which is fastest depends on
the model's register and instruction load, the stencil and the grid.  The
first fused run of a configuration times every candidate for a few launches
on scratch copies of the model's arrays (no effect on the model, its
trackers or its stimuli) and caches the winner in a JSON file keyed by the
GPU name, the model, the stencil and the grid's size class (power of two
of the node count).

The cache lives in ``$FWGPU_AUTOTUNE_CACHE`` or
``~/.cache/finitewave_gb300/autotune.json``.
"""
import ctypes
import json
import math
import os
import threading

import torch

from . import _ffi

_lock = threading.Lock()
_memo = {}

# (fused_variant, fused_k) candidates; variants 3 and 4 where the TMA kernels
# can run (packed weights; rows of a multiple of 16 nodes, or padded copies of
# the arrays).  Variants 5, 6 and 7 are
# not candidates: each was measured slower than variant 3 on the 4096^2
# Aliev-Panfilov workload (weights formed on chip, two-wide float32
# instructions, the row-marching wavefront) and is kept as an explicit
# choice only.
_TMA = [(3, 2), (3, 3), (3, 4), (3, 8), (4, 2), (4, 4), (4, 8)]
_CPASYNC = [(1, 2), (1, 4), (1, 8), (2, 2), (2, 4), (2, 8)]


def cache_path():
    return os.environ.get("FWGPU_AUTOTUNE_CACHE") or os.path.join(
        os.path.expanduser("~"), ".cache", "finitewave_gb300",
        "autotune.json")


def _load():
    try:
        with open(cache_path()) as f:
            return json.load(f)
    except (OSError, ValueError):
        return {}


def _store(table):
    path = cache_path()
    try:
        os.makedirs(os.path.dirname(path), exist_ok=True)
        tmp = path + ".tmp%d" % os.getpid()
        with open(tmp, "w") as f:
            json.dump(table, f, indent=1, sort_keys=True)
        os.replace(tmp, path)
    except OSError:
        pass   # an unwritable cache only costs a re-tune


def key(model):
    shape = model._shape()
    n = 1
    for s in shape:
        n *= s
    dev = model._device()
    name = torch.cuda.get_device_name(dev)
    parts = [name, type(model).__name__, str(model.stencil.kind),
             "%dD" % len(shape), "2^%d" % int(math.log2(max(n, 1)))]
    if len(shape) == 2 and shape[1] % 16:
        # the TMA kernels run on padded copies, where the model may keep any
        parts.append("ragged" if model._pad_ok() else "ragged flat")
    return "|".join(parts)


def _time_candidate(model, args, variant, k, steps, stream, reps=3):
    args.fused_variant = variant
    args.fused_k = k
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    # one warm-up segment, then the fastest of `reps` timed ones
    _ffi.call("fw_step", ctypes.byref(args), 0, steps, stream.cuda_stream)
    best = float("inf")
    for _ in range(reps):
        e0.record(stream)
        _ffi.call("fw_step", ctypes.byref(args), 0, steps, stream.cuda_stream)
        e1.record(stream)
        e1.synchronize()
        best = min(best, e0.elapsed_time(e1))
    return best


def tune(model, steps=96):
    """Time every fused candidate for `model` (initialised, fused form) on
    scratch copies of its arrays; returns {"variant": v, "k": k, "ms": {...}}
    and, where padded copies were timed, "flat" (the best choice on the
    model's own arrays) and "pad_from" (the steps in which the copies in and
    out are made up for).
    """
    saved = model.autotune
    model.autotune = False
    try:
        a = model._bare_args()
    finally:
        model.autotune = saved
    keep = []
    for i in range(2):
        c = model._dev["u" if i == 0 else "u_new"].clone()
        keep.append(c)
        a.u[i] = c.data_ptr()
    for i, name in enumerate(model._state_names):
        c = model._dev[name].clone()
        keep.append(c)
        a.state[i] = c.data_ptr()
        c = model._dev[name].clone()
        keep.append(c)
        a.state_b[i] = c.data_ptr()
    a.form = _ffi.FORM_FUSED
    stream = torch.cuda.current_stream()
    tma_ok = a.weights_packed and model._shape()[1] % 16 == 0
    cands = (_TMA if tma_ok else []) + _CPASYNC
    times = {}
    for v, k in cands:
        try:
            times["%d/%d" % (v, k)] = _time_candidate(model, a, v, k, steps,
                                                      stream)
        except _ffi.FwError:
            continue
    # rows that are no multiple of 16 nodes: the TMA kernels on row-padded
    # copies of the arrays, the copies in and out counted once in `steps`
    # steps (777 x 1011 nodes: 39 us, 2500 x 2501 93 us; Aliev-Panfilov
    # 2500 x 2501 takes 28.0 us a step so, 36.3 on its own arrays, 500 x 501
    # 2.7 against 2.0)
    flat = min(times, key=times.get)
    cost = dict(times)
    pad_from = 0
    mir = None
    if model._shape()[1] % 16 and model._pad_ok():
        mir = model._padded()
    if mir is not None:
        copies = _time_copies(model, mir, stream)
        mir.apply(a)
        for v, k in _TMA:
            try:
                t = _time_candidate(model, a, v, k, steps, stream)
            except _ffi.FwError:
                continue
            times["%d/%d" % (v, k)] = t
            cost["%d/%d" % (v, k)] = t + copies
    del keep
    best = min(cost, key=cost.get)
    if mir is not None:
        if best == flat:
            model._pad = None    # nothing will use the copies
        else:
            pad_from = math.ceil(copies * steps / (times[flat] - times[best]))
    v, k = (int(x) for x in best.split("/"))
    fv, fk = (int(x) for x in flat.split("/"))
    return {"variant": v, "k": k, "flat": [fv, fk], "pad_from": pad_from,
            "ms": times, "steps": steps}


def _time_copies(model, mir, stream, reps=3):
    """ms of moving a model's state into its padded copies and, unchanged,
    out again."""
    best = float("inf")
    for _ in range(reps):
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        mir.run_copies(mir.copies_in(model), stream.cuda_stream)
        mir.run_copies(mir.copies_out(model), stream.cuda_stream)
        e1.record(stream)
        e1.synchronize()
        best = min(best, e0.elapsed_time(e1))
    return best


def flat(model):
    """((fused_variant, fused_k), steps): the fastest candidate on the model's
    own arrays (rows of any length), and the number of steps from which a
    chosen TMA kernel on padded copies is faster (0: not measured)."""
    r = _entry(model)
    return tuple(r.get("flat") or (r["variant"], r["k"])), r.get("pad_from", 0)


def choose(model):
    """(fused_variant, fused_k) for `model`: from the cache, else tuned now
    and cached."""
    r = _entry(model)
    return r["variant"], r["k"]


def _entry(model):
    kk = key(model)
    with _lock:
        if kk in _memo:
            return _memo[kk]
        table = _load()
        if kk in table:
            _memo[kk] = table[kk]
            return table[kk]
    r = tune(model)
    kk = key(model)    # a model that found no room for copies has another
    with _lock:
        _memo[kk] = r
        table = _load()
        table[kk] = r
        _store(table)
    return r
