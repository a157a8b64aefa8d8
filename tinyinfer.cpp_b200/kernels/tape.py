"""Launches of one layer, recorded and repeated for the layers like it.

A step of a new shape runs eagerly, and its layers ask the kernel set for the same launches one after the other: the same
entry points with the same sizes, only over other weights and other pages.  Choosing and issuing them in Python costs 13 to
18 us a launch, several times what the launch itself takes.  So the second of a run of alike layers is run in Python with its
calls recorded, and the layers behind it repeat them natively (``ti_tape_run``) with the pointers to what a layer owns
replaced.  The first layer is not the one recorded because it has no layer in front of it whose last product waits to be added
(``_pending_runs``).

What makes a recording valid: every launch went through an entry point that has a taped form (else the number of launches and
of recorded calls differ), no torch operation but allocations and views took place, nothing is held back at the layer's end
that was not held back at its start, and the layers agree in everything that their launches may depend on (``own_layout`` of
parts/base.py) but the contents of their tensors, whose addresses, and those inside them, are replaced.  A recording
lives for one pass and holds the tensors allocated under it until the pass has issued its last launch.
"""
from __future__ import annotations

import ctypes
from bisect import bisect

import torch
from torch.overrides import TorchFunctionMode

_LAST = 1 << 64

# what a layer may ask of a tensor, and views of it: nothing of these runs on the device
_QUESTIONS = {"data_ptr", "stride", "is_contiguous", "numel", "size", "dim", "element_size", "__get__", "__len__", "__hash__",
              "view", "unflatten"}


class _Allocations(TorchFunctionMode):
    """Keeps every tensor that is allocated under it and notices any other operation on data.  (A function mode: a dispatch
    mode would bring some 900 modules with its first use, 3 to 5 s.)"""

    def __init__(self):
        super().__init__()
        self.held: list = []
        self.pure = True

    def __torch_function__(self, func, types, args=(), kwargs=None):
        out = func(*args, **(kwargs or {}))
        name = getattr(func, "__name__", "")
        if name not in _QUESTIONS:
            if func is torch.empty or func is torch.empty_like:
                self.held.append(out)
            else:
                self.pure = False
        return out


class _Tap:
    """A kernel library whose launches are recorded on their way."""

    def __init__(self, lib, calls: list):
        self._lib, self._calls = lib, calls

    def __getattr__(self, name):
        found = getattr(self._lib, name)
        taped = getattr(self._lib, name + "_taped", None)
        if taped is not None:
            fn, calls, lib = found, self._calls, self._lib
            address = ctypes.cast(taped, ctypes.c_void_p).value

            def found(*args):
                calls.append((address, lib, fn.argtypes, args))
                return fn(*args)
        setattr(self, name, found)
        return found


def _slot(kind, value) -> int:
    if kind is ctypes.c_float:
        return int.from_bytes(bytes(ctypes.c_float(value)), "little")        # rounds as a direct call does, to infinity too
    return value & 0xFFFFFFFFFFFFFFFF


def alike(layers):
    """The addresses of the layers' own tensors, a list a layer; None: the tensors differ in something that launches depend on
    (or are none)."""
    try:
        like = [(t.dtype, t.shape, t.stride(), t.is_contiguous(), t.data_ptr() % 32, getattr(t, "_ti_interleaved", None))
                for t in layers[0]]
        addresses = [[t.data_ptr() for t in layer] for layer in layers]
        for layer, mine in zip(layers[1:], addresses[1:]):
            if len(mine) != len(like):
                return None
            for t, at, (dtype, shape, strides, dense, place, interleaved) in zip(layer, mine, like):
                if (t.dtype is not dtype or at % 32 != place or t.shape != shape or t.is_contiguous() is not dense
                        or (not dense and t.stride() != strides) or getattr(t, "_ti_interleaved", None) is not interleaved):
                    return None
    except AttributeError:
        return None
    return addresses


def _inside(in_order, value):
    """(index, offset) of the tensor that the address lies in; None: in none of them."""
    at = bisect(in_order, (value, _LAST, 0)) - 1
    start, end, i = in_order[at]
    return (i, value - start) if at >= 0 and value < end else None


def record(ops, run, mine):
    """Runs one layer through ``run()`` and returns its launches as ``replay(layers)``, which takes the addresses of the own
    tensors of each layer to repeat them for (in the order of ``mine``, this layer's); None if they cannot be repeated."""
    calls: list = []
    start = ops._pending_runs
    had_more = ops._pending is not None or ops._pending_pair is not None
    libs = {"core": ops.core, "bf16": ops.__dict__.get("bf16")}
    issued = ops.issued
    with _Allocations() as watch:
        try:
            for name, lib in libs.items():
                if lib is not None:
                    ops.__dict__[name] = _Tap(lib, calls)
            run()
        finally:
            for name, lib in libs.items():
                if lib is not None:
                    ops.__dict__[name] = lib
    end = ops._pending_runs
    if (not watch.pure or had_more or ops._pending is not None or ops._pending_pair is not None
            or (start is None) != (end is None) or len(calls) != ops.issued - issued):
        return None
    renamed = {}
    if start is not None:                  # the runs that the layer in front left, and those that this one leaves
        if start[1:2] != end[1:2] or start[2] is not end[2] or start[3] != end[3]:
            return None
        renamed[start[0].data_ptr()] = end[0].data_ptr()
    in_order = []
    for i, t in enumerate(mine):
        n = t.numel() if t.is_contiguous() else 1 + sum((n - 1) * s for n, s in zip(t.shape, t.stride()))
        in_order.append((t.data_ptr(), t.data_ptr() + t.element_size() * n, i))
    in_order.sort()
    if any(after[0] < before[1] for before, after in zip(in_order, in_order[1:])):
        return None                        # an address may stand for either of two tensors
    place = {}                             # pointer -> where it lies in the layer's own tensors (None: elsewhere)
    first, slots, patches, sources = [], [], [], []
    pointer = ctypes.c_void_p
    for _, _, kinds, args in calls:
        if kinds is None or len(kinds) != len(args):
            return None
        first.append(len(slots))
        for kind, value in zip(kinds, args):
            if kind is not pointer:
                slots.append(_slot(kind, value))
            elif not value:
                slots.append(0)
            else:
                if value not in place:
                    place[value] = _inside(in_order, value)
                if place[value] is not None:
                    patches.append(len(slots))
                    sources.append(place[value])
                slots.append(renamed.get(value, value))
    n = len(calls)
    packed = ((ctypes.c_void_p * n)(*[c[0] for c in calls]), (ctypes.c_int * n)(*first), n,
              (ctypes.c_ulonglong * max(1, len(slots)))(*slots), (ctypes.c_int * max(1, len(patches)))(*patches), len(patches))

    def replay(layers):
        values = [own[i] + offset for own in layers for i, offset in sources]
        rc = ops.core.ti_tape_run(*packed, (ctypes.c_ulonglong * max(1, len(values)))(*values), len(layers))
        ops.launches += n * len(layers)
        ops.issued += n * len(layers)
        return None if rc == 0 else calls[rc - 1][1]
    replay.held = (watch.held, start)      # alive until the last launch has been issued
    return replay
