"""Launch-shape autotuner front end with a JSON cache.

smpc_autotune (C ABI) times every launch-shape variant of the fast-path
solvent-binning, collide and MD kernels (and of the periodic MD, in contexts
with periodic boxes) on the context's own workload with CUDA events, keeps the
fastest and restores the state its trial cycles advanced. This module caches
the choice per GPU model, workload signature and kernel sources, so later runs
of the same workload start tuned, and kernels that have changed are measured
again.
"""
from __future__ import annotations

import functools
import hashlib
import json
import os
from typing import Optional

HERE = os.path.dirname(os.path.abspath(__file__))
CACHE = os.path.join(HERE, "_tune", "autotune_cache.json")


def gpu_name() -> str:
    try:
        import torch
        if torch.cuda.is_available():
            return torch.cuda.get_device_name(0)
    except Exception:  # torch is optional here
        pass
    return "unknown-gpu"


@functools.lru_cache(maxsize=None)
def kernels_id(folder: str = os.path.join(HERE, "csrc")) -> str:
    """Digest of the kernel sources: what was fastest among other kernels need not be now."""
    h = hashlib.sha256()
    for name in sorted(n for n in os.listdir(folder) if n.endswith((".cu", ".cuh", ".h"))):
        with open(os.path.join(folder, name), "rb") as f:
            h.update(name.encode() + b"\0" + f.read() + b"\0")
    return h.hexdigest()[:12]


def signature(n_rep: int, particles: int, cells: int, monomers: int) -> str:
    return (f"{gpu_name()}|rep={n_rep}|particles={particles}|cells={cells}|monomers={monomers}"
            f"|kernels={kernels_id()}")


def _load(path: str) -> dict:
    try:
        with open(path) as f:
            return json.load(f)
    except (OSError, ValueError):
        return {}


def tune(ctx, key: str, cycles: int = 3, cache_path: Optional[str] = None,
         force: bool = False) -> dict:
    """Applies the cached variants for `key`, or measures and caches them."""
    path = cache_path or CACHE
    cache = _load(path)
    if not force and key in cache:
        index = cache[key]["index"]
        ctx.set_variants(*index[:3])
        if len(index) > 3:
            ctx.set_pmd_variant(index[3])
        return dict(cache[key], cached=True)
    report = ctx.autotune(cycles)
    entry = {"index": list(ctx.get_variants()) + [ctx.get_pmd_variant()], "report": report}
    cache[key] = entry
    os.makedirs(os.path.dirname(path), exist_ok=True)
    tmp = path + ".tmp%d" % os.getpid()
    with open(tmp, "w") as f:
        json.dump(cache, f, indent=1, sort_keys=True)
    os.replace(tmp, path)
    return dict(entry, cached=False)
