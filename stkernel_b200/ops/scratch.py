"""Per-device scratch arena with cached, address-stable views.

Each named buffer is allocated once per device and only grows, so a kernel
launched with the same name and size sees the same address every step (needed
for CUDA-graph replay).  Buffers used on different streams must use different
names: two names never alias; inside `side_branch(stream)` every name gets the
branch's suffix, so the same op may run on the main and on a side stream at once.
This is the engine's equivalent of the reference's eager scratch pool
(overlay/eager_scratch.py:27-168).
"""
from __future__ import annotations

from contextlib import contextmanager
from typing import Dict, List, Sequence, Tuple

import torch

_pool: Dict[Tuple[str, str], torch.Tensor] = {}
# The view handed out last under each name: (shape, dtype, buffer, view, its place in the pool).  Steps ask for the same shapes again
# and again, and cutting a view anew costs 9.6 us of Python against 0.5 us for finding this one; a view holds no memory of its own,
# and one per name is kept.  None is an inference tensor, which calls outside of inference mode may not write to, and one that has become
# part of an autograd graph is not handed out again.
_views: Dict[tuple, tuple] = {}
# buffers that were outgrown: captured graphs may still hold their addresses
_outgrown: List[torch.Tensor] = []
_frozen = False
_branch = ""


@contextmanager
def side_branch(stream, label: str = "side"):
    """Run the enclosed ops on `stream` (a fork of the step's dependency graph, also under CUDA-graph capture) with
    their own copies of every named scratch buffer.  The caller orders the streams with events."""
    global _branch
    prev = _branch
    _branch = "@" + label
    try:
        with torch.cuda.stream(stream):
            yield
    finally:
        _branch = prev


def freeze(flag: bool = True) -> None:
    """After freezing (graphs captured) a request that would grow a buffer raises instead."""
    global _frozen
    _frozen = flag


def scratch(name: str, shape: Sequence[int], dtype: torch.dtype, device, zero: bool = False) -> torch.Tensor:
    shape = tuple(shape)
    place = (name, _branch, device)
    last = _views.get(place)
    if last is not None and last[0] == shape and last[1] is dtype and _pool.get(last[4]) is last[2] and not last[3].requires_grad:
        return last[3]
    if torch.is_inference_mode_enabled():
        with torch.inference_mode(False):
            return _cut(name, shape, dtype, device, zero, place)
    return _cut(name, shape, dtype, device, zero, place)


def _cut(name: str, shape: tuple, dtype: torch.dtype, device, zero: bool, place: tuple) -> torch.Tensor:
    n = 1
    for d in shape:
        n *= int(d)
    used = n * dtype.itemsize
    nbytes = max(used, 16)
    key = (name + _branch, str(device))
    buf = _pool.get(key)
    if buf is None or buf.numel() < nbytes:
        if _frozen and buf is not None:
            raise RuntimeError(f"scratch buffer {name!r} would grow after graphs were captured")
        cap = max(nbytes, 2 * buf.numel() if buf is not None else 0)
        cap = (cap + 255) // 256 * 256
        if buf is not None:
            _outgrown.append(buf)
        buf = torch.zeros(cap, dtype=torch.uint8, device=device) if zero else torch.empty(cap, dtype=torch.uint8, device=device)
        _pool[key] = buf
    view = buf[:used].view(dtype).view(*shape)
    _views[place] = (shape, dtype, buf, view, key)
    return view


def reset() -> None:
    _pool.clear()
    _views.clear()
    _outgrown.clear()


def total_bytes() -> int:
    return sum(b.numel() for b in list(_pool.values()) + _outgrown)
