"""Measured choice of the psi sweep's launch shape, persisted per problem.

The FP32 psi sweep has two kernels: the cooperative loop (the default; its strip
height follows from the size) and the bulk-copy ring, compiled for the heights in
``STRIP_ROWS``; FP64 has one without strips.  By default a handle takes the loop, and
for the ring the height an item-count model picks.  ``tune(handle)`` measures instead:
it times one sweep launch (``glgpu_time_sweeps``: CUDA events, L2 flushed
before each launch) for every (kernel, height) pair, applies the fastest, and
stores it in a JSON cache keyed by (dtype, Nx, Ny, kappa finite, kernel set), so that
later handles with the same key take the stored choice without measuring.  (The heights
make no difference to kernel 0.)  Domains that fit on chip run no sweep kernel but the
resident loop, which selecting kernel 1 would switch off: they keep kernel 0 whatever the
sweeps measure.  Results do not depend on the choice: every pair computes the same values
bitwise (tests/test_gpu_strip_rows.py, tests/test_gpu_psi_kernels.py).

The cache file is ``$SVIRL_GB300_TUNE_CACHE`` or ``~/.cache/svirl_gb300/psi_sweep.json``.
No counterpart in the reference, whose kernels have one fixed launch shape
(128-thread blocks, svirl/parallel/startup.py:65).
"""
import json
import os

import numpy as np

STRIP_ROWS = (8, 12, 17)  # the heights libglgpu compiles the sweep for
KERNELS_FP32 = (0, 1)     # 0 cooperative loop, 1 bulk-copy ring (glgpu_set_psi_sweep_kernel)
KERNEL_SET = 2            # of the key: choices among other kernels than these are not taken over


def cache_path():
    p = os.environ.get("SVIRL_GB300_TUNE_CACHE")
    if p:
        return p
    return os.path.join(os.path.expanduser("~"), ".cache", "svirl_gb300", "psi_sweep.json")


def key_of(handle):
    return "%s:%dx%d:%s:%d" % (np.dtype(handle.dtype).name, handle.Nx, handle.Ny,
                               "finite" if handle.kappa_finite() else "inf", KERNEL_SET)


def _load(path):
    try:
        with open(path) as fh:
            return json.load(fh)
    except (OSError, ValueError):
        return {}


def _store(path, table):
    d = os.path.dirname(path)
    if d:
        os.makedirs(d, exist_ok=True)
    tmp = path + ".tmp"
    with open(tmp, "w") as fh:
        json.dump(table, fh, indent=1, sort_keys=True)
    os.replace(tmp, path)


def apply(handle, choice):
    handle.set_psi_sweep_kernel(int(choice["kernel"]))
    handle.set_psi_strip_rows(int(choice["rows"]))


def tune(handle, reps=5, path=None, force=False):
    """Measure (or look up) and apply the fastest psi sweep launch shape for
    `handle`; returns the choice {"kernel", "rows", "us", "measured": {...}}."""
    path = path or cache_path()
    table = _load(path)
    key = key_of(handle)
    on_chip = getattr(handle, "td_resident", lambda: False)()
    if not force and key in table:
        choice = dict(table[key], cached=True)
        if on_chip:
            choice["kernel"] = 0
        apply(handle, choice)
        return choice
    kernels = KERNELS_FP32 if np.dtype(handle.dtype) == np.float32 else (0,)
    measured = {}
    for kern in kernels:
        for rows in STRIP_ROWS:
            handle.set_psi_sweep_kernel(kern)
            handle.set_psi_strip_rows(rows)
            handle.time_sweeps(0, 1)  # warm-up launch
            measured["%d/%d" % (kern, rows)] = 1e3 * handle.time_sweeps(0, reps)
    best = min((k for k in measured if not on_chip or k.startswith("0/")), key=measured.get)
    kern, rows = (int(x) for x in best.split("/"))
    choice = {"kernel": kern, "rows": rows, "us": measured[best], "measured": measured}
    apply(handle, choice)
    table[key] = choice
    _store(path, table)
    return dict(choice, cached=False)
