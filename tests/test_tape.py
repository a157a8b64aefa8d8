"""What makes a layer's recorded launches valid for the layers like it: parts whose class itself says so, equal in everything but
their tensors; the addresses of those tensors, and addresses inside them, are the layer's own in every repetition.  A kernel set
whose entry points note their pointers stands for the device."""
import ctypes
import threading
from types import SimpleNamespace

import pytest
import torch

from tinyinfer_b200.config import PartSpec
from tinyinfer_b200.kernels import tape
from tinyinfer_b200.parts.attention import Attention
from tinyinfer_b200.parts.base import own_layout, own_tensors
from tinyinfer_b200.parts.block import PreNormBlock
from tinyinfer_b200.parts.mlp import SwiGLU
from tinyinfer_b200.parts.norm import RMSNorm


class NotingLib:
    """One entry point, ``ti_x(pointer, number)``, and the native repetition of its calls."""

    def __init__(self):
        self.seen, self.lock = [], threading.Lock()
        self.ti_x_taped = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p)(lambda slots: 0)

        def ti_x(pointer, number):
            self.seen.append((pointer, number))
            return 0
        ti_x.argtypes = [ctypes.c_void_p, ctypes.c_int]
        self.ti_x = ti_x

    def ti_tape_run(self, calls, first, num_calls, slots, patch_slot, num_patches, values, layers):
        for layer in range(layers):
            for p in range(num_patches):
                slots[patch_slot[p]] = values[layer * num_patches + p]
            for c in range(num_calls):
                self.seen.append((slots[first[c]], slots[first[c] + 1]))
        return 0


def _ops():
    ops = SimpleNamespace(core=NotingLib(), _pending_runs=None, _pending=None, _pending_pair=None, issued=0, launches=0, use_tape=True)

    def x(pointer, number):
        ops.issued += 1
        ops.core.ti_x(pointer, number)
    ops.x = x
    return ops


class Plain(SwiGLU):
    """Reads its two matrices, one of them from an address inside it."""
    launches_repeat = True

    def __init__(self):
        super().__init__(8, 16)
        self.w_gate_up, self.w_down = torch.zeros(32, 8), torch.zeros(8, 16)

    def forward(self, ops, h, residual, step):
        ops.x(self.w_gate_up.data_ptr(), 1)
        ops.x(self.w_gate_up[16:].data_ptr() if step is None else self.w_gate_up.data_ptr() + 16 * 8 * 4, 2)
        ops.x(self.w_down.data_ptr(), 3)


class Adapted(Plain):
    """One tensor more, as a class outside the package would add it, without a word on its launches."""

    def __init__(self):
        super().__init__()
        self.adapter = torch.zeros(4, 8)

    def forward(self, ops, h, residual, step):
        super().forward(ops, h, residual, step)
        ops.x(self.adapter.data_ptr(), 4)


class AdaptedAndSaid(Adapted):
    launches_repeat = True


def _run(layers):
    from tinyinfer_b200.kernels.cuda_ops import CudaOps
    ops = _ops()

    layout = own_layout(layers[0])

    def own(k):
        tensors = []
        return tensors if layout and own_tensors(layers[k], layout, tensors) else None
    before = len(ops.core.seen)
    CudaOps.repeat_layers(ops, len(layers), lambda k: layers[k].forward(ops, None, None, True), own)
    got = ops.core.seen[before:]
    python = ops.issued
    ops.core.seen.clear()
    for layer in layers:
        layer.forward(ops, None, None, True)
    return got, list(ops.core.seen), python


@pytest.mark.parametrize("part", [Plain, Adapted, AdaptedAndSaid])
def test_every_layer_reads_its_own_tensors(part):
    got, want, python = _run([part() for _ in range(6)])
    assert got == want
    per_layer = len(want) // 6
    assert part is Adapted or python == 6 * per_layer      # launches are counted, repeated ones too


def test_classes_speak_for_themselves_alone():
    assert own_layout(Plain()) and own_layout(AdaptedAndSaid())
    assert own_layout(Adapted()) is None
    tensors = []
    assert own_tensors(AdaptedAndSaid(), own_layout(AdaptedAndSaid()), tensors) and len(tensors) == 3
    assert not own_tensors(Adapted(), own_layout(Plain()), []) and not own_tensors(AdaptedAndSaid(), own_layout(Plain()), [])
    part = Plain()
    part.forward = lambda *a: None                          # a method replaced on one part
    assert own_layout(part) is None and not own_tensors(part, own_layout(Plain()), [])
    part = Plain()
    part.table = {"a": torch.zeros(1)}                      # tensors out of sight
    assert own_layout(part) is None and not own_tensors(part, own_layout(Plain()), [])
    part = Plain()
    del part.w_down
    assert not own_tensors(part, own_layout(Plain()), [])


def _block(**changed):
    position = PartSpec("rope_neox", {"head_dim": 16, "theta": 1e4})
    mixer = Attention(hidden_size=64, num_heads=4, num_kv_heads=2, head_dim=16, qk_norm_eps=1e-6, position=position)
    block = PreNormBlock(mixer, RMSNorm(64, 1e-6), SwiGLU(64, 96), RMSNorm(64, 1e-6))
    mixer.w_qkv, mixer.w_o, mixer.q_norm, mixer.k_norm = (torch.zeros(n, 4) for n in (8, 4, 2, 2))
    block.ffn.w_gate_up, block.ffn.w_down = torch.zeros(8, 4), torch.zeros(4, 4)
    block.mixer_norm.weight, block.ffn_norm.weight = torch.zeros(4), torch.zeros(4)
    for path, value in changed.items():
        *way, name = path.split("__")
        at = block
        for w in way:
            at = getattr(at, w)
        setattr(at, name, value)
    return block


def _alike(other):
    tensors = [[], []]
    layout = own_layout(_block())
    if not all(own_tensors(b, layout, t) for b, t in zip((_block(), other), tensors)):
        return None
    assert len(tensors[0]) == 8
    return tape.alike(tensors)


def test_the_parts_of_a_layer_are_seen_through():
    other = _block()
    assert _alike(other)[1] == [t.data_ptr() for t in (
        other.mixer.w_qkv, other.mixer.w_o, other.mixer.q_norm, other.mixer.k_norm, other.ffn.w_gate_up, other.ffn.w_down,
        other.mixer_norm.weight, other.ffn_norm.weight)]


@pytest.mark.parametrize("changed", [{"mixer__scale": 0.5}, {"mixer_norm__eps": 1e-3}, {"mixer__position__theta": 3e4},
                                     {"ffn__w_down": torch.zeros(4, 4, dtype=torch.bfloat16)}, {"mixer__window": 7},
                                     {"ffn__factor": 2.0}, {"mixer__w_o": None}])
def test_layers_that_differ_in_anything_but_contents_are_told_apart(changed):
    assert _alike(_block(**changed)) is None


def test_tensors_that_overlap_are_not_repeated():
    class Two(Plain):
        launches_repeat = True

        def __init__(self):
            super().__init__()
            self.w_second = self.w_gate_up[8:]
    made = []
    real = tape.record
    try:
        tape.record = lambda *a: made.append(real(*a)) or made[-1]
        got, want, _ = _run([Two() for _ in range(5)])
    finally:
        tape.record = real
    assert got == want and made == [None]


def test_numbers_are_handed_on_as_a_direct_call_hands_them_on():
    for value in (0.1, -3, 1e39, -1e39, 1e-46, float("inf")):
        bits = tape._slot(ctypes.c_float, value)
        assert ctypes.c_float.from_buffer_copy(bits.to_bytes(4, "little")).value == ctypes.c_float(value).value
    assert tape._slot(ctypes.c_int, -2) == 2 ** 64 - 2 and tape._slot(ctypes.c_int, True) == 1
