"""Prompt portions of the attention with options on tcgen05, against float64 and beside the mma.sync kernel: rows of one
to nine chunks of 64 elements (one that ends inside a chunk), values of one to eight, one and two slices, groups that fill
the 128 rows of a block and that do not, tiles of keys that end before, at and behind an edge, pages of one to four runs
a tile, requests of one token beside portions, and every option."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from tinyinfer_b200.kernels import CudaOps
    return CudaOps(DEV)


def _attend(q, k, v, pos, scale, opt, head_scale, sink):
    group = q.shape[1] // k.shape[1]
    k, v = (x.repeat_interleave(group, 1) for x in (k, v))
    s = torch.einsum("thd,shd->hts", q, k) * scale
    if head_scale is not None:
        s = s * head_scale[:, None, None]
    if opt.get("cap"):
        s = opt["cap"] * torch.tanh(s / opt["cap"])
    key = torch.arange(k.shape[0], device=q.device)
    dark = key[None] > pos[:, None]
    if opt.get("window"):
        dark |= key[None] <= pos[:, None] - opt["window"]
    if opt.get("chunk"):
        dark |= key[None] // opt["chunk"] != pos[:, None] // opt["chunk"]
    s = s.masked_fill(dark, -torch.inf)
    if sink is not None:
        s = torch.cat([s, sink[:, None, None].expand(-1, s.shape[1], 1)], 2)
    return torch.einsum("hts,shd->thd", torch.softmax(s, -1)[..., :k.shape[0]], v)


@pytest.mark.parametrize("heads,kv,dk,dv,shared,page", [
    (16, 1, 576, 512, True, 64), (16, 1, 288, 256, True, 64), (24, 1, 96, 64, True, 16), (5, 1, 320, 192, True, 48),
    (32, 1, 576, 512, True, 32), (4, 1, 512, 512, True, 64), (40, 1, 256, 256, True, 16), (4, 1, 64, 64, True, 64),
    (16, 4, 64, 64, False, 64), (16, 4, 128, 128, False, 64), (6, 2, 128, 128, False, 16), (3, 3, 64, 64, False, 48)])
@pytest.mark.parametrize("opt", [
    {}, {"window": 70}, {"chunk": 150, "cap": 4.0, "head_scale": True, "gate": "head"}, {"sink": True, "gate": "element"}])
def test_portions(ops, monkeypatch, heads, kv, dk, dv, shared, page, opt):
    from tinyinfer_b200.kernels.step_lists import option_tiles, row_tiles
    # contexts that end before, at and behind a tile of keys; a long one behind a portion of few tokens
    ctx, new = [64, 1, 65, 400, 63, 200, 130], [64, 1, 65, 140, 3, 1, 2]
    g = torch.Generator(device=DEV).manual_seed(dk + dv + heads)
    ti = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    blocks = [-(-c // page) for c in ctx]
    order = torch.randperm(sum(blocks) + 2, generator=torch.Generator().manual_seed(3)).tolist()
    table = torch.full((len(ctx), max(blocks)), -1, dtype=torch.int32)
    keys = [rnd(c, kv, dk).bfloat16() for c in ctx]
    values = [k[:, :, :dv] for k in keys] if shared else [rnd(c, kv, dv).bfloat16() for c in ctx]
    pages = torch.zeros((sum(blocks) + 2, kv * page * (dk if shared else dk + dv)), dtype=torch.bfloat16, device=DEV)
    for r, c in enumerate(ctx):
        for b in range(blocks[r]):
            table[r, b] = order.pop()
            n = min(page, c - b * page)
            at = pages[table[r, b]]
            at[:kv * page * dk].view(kv, page, dk)[:, :n] = keys[r][b * page:b * page + n].transpose(0, 1)
            if not shared:
                at[kv * page * dk:].view(kv, page, dv)[:, :n] = values[r][b * page:b * page + n].transpose(0, 1)
    starts = [c - n for c, n in zip(ctx, new)]
    positions = [p for s, c in zip(starts, ctx) for p in range(s, c)]
    t, group = len(positions), heads // kv
    gp = ops._group_rows(heads, kv)
    lists = {f"row_tiles_{64 // gp}": ti(row_tiles(new, starts, 64 // gp).tolist()).view(-1, 3),
             f"option_tiles_{128 // group}": ti(option_tiles(new, starts, 128 // group).tolist()).view(-1, 3)}
    step = SimpleNamespace(positions=ti(positions), req_of_tok=ti([r for r, n in enumerate(new) for _ in range(n)]),
                           scratch={}, lists=lists, max_position=max(ctx), max_ctx_len=max(ctx), max_q_len=max(new))
    cache = SimpleNamespace(pages=pages, block_table=table.to(DEV), page_size=page, writes=True)
    q = rnd(t, heads, dk).bfloat16()
    head_scale = 1 + rnd(heads).abs() if opt.get("head_scale") else None
    sink = rnd(heads) + 1.0 if opt.get("sink") else None
    gate = rnd(t, heads if opt["gate"] == "head" else heads * dv) if opt.get("gate") else None
    scale = 2.0 * dk ** -0.5
    assert ops.mixers_tc.ti_attn_options_umma_tokens(dk, dv, page, int(shared), heads, kv) == 128 // group
    outs = []
    for umma in (True, False):
        monkeypatch.setattr(ops, "use_umma_attention_options", umma)
        out = torch.full((t, heads * dv), 9.0, dtype=torch.bfloat16, device=DEV)
        ops.attention_options(q.view(t, -1), step, cache, out, heads, kv, dk, dv, scale, window=opt.get("window"),
                              chunk=opt.get("chunk"), softcap=opt.get("cap"), head_scale=head_scale, sink=sink, gate=gate,
                              gate_per_head=opt.get("gate") == "head", shared_rows=shared)
        outs.append(out.double().view(t, heads, dv))
    ops.check_status()
    at, far = 0, [0.0, 0.0]
    for r, n in enumerate(new):
        d = lambda x: None if x is None else x.double()
        want = _attend(q[at:at + n].double(), keys[r].double(), values[r].double(), step.positions[at:at + n].long(), scale,
                       opt, d(head_scale), d(sink))
        if gate is not None:
            want = want * torch.sigmoid(gate[at:at + n].double()).view(n, heads, -1)
        for i, out in enumerate(outs):
            diff = (out[at:at + n] - want).abs()
            # half a unit of bfloat16, and float32 scores of size dk that shift a weight by some 1e-5
            assert bool((diff <= want.abs() * 2.0 ** -8 + 1e-4).all()), (r, i, float(diff.max()))
            far[i] += float((diff ** 2).sum())
        at += n
    assert far[0] <= 1.05 * far[1], "further from float64 than the mma.sync kernel"
