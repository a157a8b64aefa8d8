"""Alike layers repeated from a recording give the bits that running them one by one gives, over steps of every kind: prompt
portions whose last product leaves runs to be added, mixed steps, single tokens, float32; and what cannot be repeated is not."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _config(head_dim=128, hidden=512, ff=1024):
    return dict(architectures=["Qwen3ForCausalLM"], num_hidden_layers=6, hidden_size=hidden, num_attention_heads=4,
                num_key_value_heads=2, head_dim=head_dim, intermediate_size=ff, vocab_size=512, rope_theta=10000.0,
                rms_norm_eps=1e-6, tie_word_embeddings=True, max_position_embeddings=4096)


STEPS = [[("a", 300, [299]), ("b", 70, [])], [("a", 1, [0]), ("b", 600, [5, 599])], [("a", 1, [0]), ("b", 1, [0])],
         [("c", 17, [16])], [("a", 1, [0]), ("b", 40, [39]), ("c", 1, [0])], [("c", 9, [8])]]


def _run(engine, tape):
    from tinyinfer_b200 import StepEntry
    engine.ops.use_tape = tape
    g = torch.Generator().manual_seed(2)
    for r in "abc":
        engine.add_request(r)
    outs = []
    for step in STEPS:
        entries = [StepEntry(r, torch.randint(0, 512, (n,), generator=g).tolist(), want) for r, n, want in step]
        before = engine.ops.launches
        outs.append((engine.step(entries).clone(), engine.ops.launches - before))
    for r in "abc":
        engine.finish(r)
    engine.ops.check_status()
    return outs


@pytest.mark.parametrize("dtype,kw", [("bfloat16", {}), ("bfloat16", {"head_dim": 64}), ("float32", {}),
                                      ("bfloat16", {"hidden": 1024, "ff": 3072})])
def test_repeated_layers_give_the_same_bits(dtype, kw, monkeypatch):
    from tinyinfer_b200 import Engine
    from tinyinfer_b200.kernels import tape
    engine = Engine(config=_config(**kw), seed=1, dtype=dtype, device=DEV, num_pages=64, max_requests=3)
    want = _run(engine, False)
    made = []
    real = tape.record
    monkeypatch.setattr(tape, "record", lambda *a: made.append(real(*a)) or made[-1])
    got = _run(engine, True)
    for (a, n), (b, m) in zip(want, got):
        assert torch.equal(a, b) and n == m
    assert len(made) == len(STEPS) and all(r is not None for r in made)


def test_layers_that_cannot_be_repeated_run_one_by_one(monkeypatch):
    """An operation of torch inside a layer, a weight of another type in one of them: same results, no recording used."""
    from tinyinfer_b200 import Engine
    from tinyinfer_b200.kernels import tape
    engine = Engine(config=_config(), seed=1, dtype="bfloat16", device=DEV, num_pages=64, max_requests=3)
    want = _run(engine, False)
    made = []
    real = tape.record
    monkeypatch.setattr(tape, "record", lambda *a: made.append(real(*a)) or made[-1])
    ops = engine.ops
    linear = ops.linear

    def touched(a, w, out, **kw):
        torch.zeros(1, device=DEV)
        return linear(a, w, out, **kw)
    monkeypatch.setattr(ops, "linear", touched)
    for (a, _), (b, _) in zip(want, _run(engine, True)):
        assert torch.equal(a, b)
    assert made and all(r is None for r in made)
    monkeypatch.undo()
    made.clear()
    monkeypatch.setattr(tape, "record", lambda *a: made.append(1))
    mixer = engine.model.blocks[3].mixer
    mixer.w_o = mixer.w_o.float()
    _run(engine, True)
    assert not made, "layers of unlike weights were recorded"


def _adapted_parts():
    """A feed-forward from outside the package: SwiGLU and one more matrix a layer."""
    from tinyinfer_b200.parts.base import MATRIX, WeightSpec
    from tinyinfer_b200.parts.mlp import SwiGLU

    class Adapted(SwiGLU):
        def weight_specs(self):
            return {**super().weight_specs(), "adapter.weight": WeightSpec((self.hidden_size, self.hidden_size), MATRIX)}

        def load_weights(self, tensors, ops):
            super().load_weights(tensors, ops)
            self.adapter = ops.pack_linear(tensors["adapter.weight"])

        def forward(self, ops, h, residual, step):
            ops.linear(h, self.adapter, residual, accumulate=True)
            super().forward(ops, h, residual, step)

    class AdaptedAndSaid(Adapted):
        launches_repeat = True
    return Adapted, AdaptedAndSaid


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("said", [False, True])
def test_parts_from_outside_the_package_read_their_own_tensors(dtype, said, monkeypatch):
    from tinyinfer_b200 import Engine
    from tinyinfer_b200.kernels import tape
    from tinyinfer_b200.parts import register_part
    from tinyinfer_b200.parts.mlp import SwiGLU
    register_part("ffn", "swiglu", _adapted_parts()[said])
    try:
        engine = Engine(config=_config(), seed=1, dtype=dtype, device=DEV, num_pages=64, max_requests=3)
    finally:
        register_part("ffn", "swiglu", SwiGLU)
    want = _run(engine, False)
    made = []
    real = tape.record
    monkeypatch.setattr(tape, "record", lambda *a: made.append(real(*a)) or made[-1])
    for (a, n), (b, m) in zip(want, _run(engine, True)):
        assert torch.equal(a, b) and n == m
    assert len(made) == (len(STEPS) if said else 0) and all(r is not None for r in made)


def test_a_number_changed_in_one_layer_is_kept(monkeypatch):
    from tinyinfer_b200 import Engine
    from tinyinfer_b200.kernels import tape
    engine = Engine(config=_config(), seed=1, dtype="bfloat16", device=DEV, num_pages=64, max_requests=3)
    plain = _run(engine, False)
    engine.model.blocks[3].mixer.scale *= 3.0
    want = _run(engine, False)
    assert not torch.equal(plain[0][0], want[0][0])
    monkeypatch.setattr(tape, "record", lambda *a: pytest.fail("layers of unlike numbers were recorded"))
    for (a, _), (b, _) in zip(want, _run(engine, True)):
        assert torch.equal(a, b)
