"""Prompt portions of the attention with options against float64 where the order of the kernel's roles matters."""
from types import SimpleNamespace

import pytest
import torch

from test_gpu_attention_options_umma import _attend

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from tinyinfer_b200.kernels import CudaOps
    return CudaOps(DEV)


def _check(ops, heads, kv, dk, dv, shared, page, ctx, new, opt={}, shape_keys=None, left=0.0, released=False, one_tile=False):
    """Attends the last ``new[r]`` of ``ctx[r]`` tokens of every request and compares every row with float64.  ``left`` fills
    what earlier requests have left in the pool (a number, or "large" for rows of random large numbers); ``released``:
    pages wholly in front of the first visible key of a request's first new token are gone from its table."""
    from tinyinfer_b200.kernels.step_lists import option_tiles, row_tiles
    g = torch.Generator(device=DEV).manual_seed(dk + dv + heads)
    ti = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    blocks = [-(-c // page) for c in ctx]
    count = sum(blocks) + 2
    order = torch.randperm(count, generator=torch.Generator().manual_seed(3)).tolist()
    table = torch.full((len(ctx), max(blocks)), -1, dtype=torch.int32)
    q = rnd(sum(new), heads, dk).bfloat16()
    keys = [rnd(c, kv, dk).bfloat16() for c in ctx]
    if shape_keys is not None:
        q, keys = shape_keys(q, keys)
    values = [k[:, :, :dv] for k in keys] if shared else [rnd(c, kv, dv).bfloat16() for c in ctx]
    pages = torch.empty((count, kv * page * (dk if shared else dk + dv)), dtype=torch.bfloat16, device=DEV)
    pages.copy_(1000.0 * rnd(*pages.shape)) if left == "large" else pages.fill_(left)
    for r, c in enumerate(ctx):
        for b in range(blocks[r]):
            table[r, b] = order.pop()
            n = min(page, c - b * page)
            at = pages[table[r, b]]
            at[:kv * page * dk].view(kv, page, dk)[:, :n] = keys[r][b * page:b * page + n].transpose(0, 1)
            if not shared:
                at[kv * page * dk:].view(kv, page, dv)[:, :n] = values[r][b * page:b * page + n].transpose(0, 1)
    starts = [c - n for c, n in zip(ctx, new)]
    if released:
        for r, start in enumerate(starts):
            first = max(0, start - opt["window"] + 1) if opt.get("window") else start // opt["chunk"] * opt["chunk"]
            pages[table[r, :first // page].long()] = float("nan")
            table[r, :first // page] = -1
    positions = [p for s, c in zip(starts, ctx) for p in range(s, c)]
    t, group = len(positions), heads // kv
    gp = ops._group_rows(heads, kv)
    lists = {f"row_tiles_{64 // gp}": ti(row_tiles(new, starts, 64 // gp).tolist()).view(-1, 3),
             f"option_tiles_{128 // group}": ti(option_tiles(new, starts, 128 // group).tolist()).view(-1, 3)}
    step = SimpleNamespace(positions=ti(positions), req_of_tok=ti([r for r, n in enumerate(new) for _ in range(n)]),
                           scratch={}, lists=lists, max_position=max(ctx), max_ctx_len=max(ctx), max_q_len=max(new),
                           one_tile=one_tile)
    cache = SimpleNamespace(pages=pages, block_table=table.to(DEV), page_size=page, writes=True)
    scale = 2.0 * dk ** -0.5
    out = torch.full((t, heads * dv), 9.0, dtype=torch.bfloat16, device=DEV)
    ops.attention_options(q.reshape(t, -1), step, cache, out, heads, kv, dk, dv, scale, window=opt.get("window"),
                          chunk=opt.get("chunk"), softcap=opt.get("cap"), shared_rows=shared)
    ops.check_status()
    at = 0
    for r, n in enumerate(new):
        want = _attend(q[at:at + n].double(), keys[r].double(), values[r].double(), step.positions[at:at + n].long(), scale,
                       opt, None, None)
        diff = (out[at:at + n].double().view(n, heads, dv) - want).abs()
        # half a unit of bfloat16, and float32 scores of size dk that shift a weight by some 1e-5
        assert bool((diff <= want.abs() * 2.0 ** -8 + 1e-4).all()), (r, float(diff.max()))
        at += n
    return out


SIZES = [(16, 1, 576, 512, True, 64), (16, 1, 288, 256, True, 64), (16, 4, 128, 128, False, 64), (16, 4, 64, 64, False, 32)]


@pytest.mark.parametrize("heads,kv,dk,dv,shared,page", SIZES)
def test_weights_replaced_without_a_new_reference(ops, heads, kv, dk, dv, shared, page):
    """A row's largest score lies in its first tile of keys, so that no later tile brings the outputs to a new reference:
    every tile's weights replace the ones before directly behind the value products that read them.  Portions of as
    many blocks as fill every SM, over some thirty tiles of keys."""
    def first_tile_wins(q, keys):
        q[:, :, 0] = 4.0                       # a common direction: the first 64 keys stand out in it, the others fall off
        for k in keys:
            k[:64, :, 0] = 3.0
            k[64:, :, 0] = torch.linspace(1.0, -1.0, k.shape[0], device=DEV)[64:, None].bfloat16()
        return q, keys
    _check(ops, heads, kv, dk, dv, shared, page, [2000, 1700, 90], [600, 500, 90], shape_keys=first_tile_wins)


@pytest.mark.parametrize("heads,kv,size,page", [(16, 4, 128, 64), (16, 4, 64, 16), (6, 6, 128, 16)])
@pytest.mark.parametrize("cap", [None, 5.0])
def test_scores_behind_the_weights_they_replace(ops, heads, kv, size, page, cap):
    """Heads with values of their own: a tile's scores come into the columns of tensor memory that hold the last part of
    the weights of the tile before.  Two blocks on every SM over an odd and an even number of tiles; repeated launches
    give the same bits."""
    outs = [_check(ops, heads, kv, size, size, False, page, [4100, 2048, 65], [1300, 1024, 65], {"cap": cap}) for _ in range(3)]
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


@pytest.mark.parametrize("heads,kv,dk,dv,shared,page", SIZES + [(24, 1, 96, 64, True, 16), (6, 2, 128, 128, False, 16)])
@pytest.mark.parametrize("left", [float("nan"), float("inf"), "large"])
@pytest.mark.parametrize("opt", [{}, {"window": 70}, {"chunk": 150, "cap": 4.0}])
def test_what_earlier_requests_left(ops, monkeypatch, heads, kv, dk, dv, shared, page, left, opt):
    """A reused page holds infinities and NaN behind a context's end, and pages that a window or a chunk has passed are
    gone: no query may see either, on tcgen05, on mma.sync, and in a step of single tokens."""
    ctx, new = [64, 1, 65, 400, 63, 200, 130, 77], [64, 1, 65, 140, 3, 1, 2, 77]
    for umma in (True, False):
        monkeypatch.setattr(ops, "use_umma_attention_options", umma)
        _check(ops, heads, kv, dk, dv, shared, page, ctx, new, opt, left=left, released=bool(opt))
    _check(ops, heads, kv, dk, dv, shared, page, ctx, [1] * len(ctx), opt, left=left, released=bool(opt))


@pytest.mark.parametrize("heads,kv,size,most", [(16, 4, 64, 8), (16, 4, 128, 2), (6, 6, 128, 8), (8, 1, 64, 4), (16, 1, 128, 0)])
def test_short_portions_in_one_tile_of_keys(ops, monkeypatch, heads, kv, size, most):
    """A step whose contexts all end in their first tile of keys takes the tcgen05 kernel for portions of more than
    ``most`` tokens; any step with a longer context takes it."""
    taken = []
    real = ops.mixers_tc.ti_attn_options_umma
    monkeypatch.setattr(ops.mixers_tc, "ti_attn_options_umma", lambda *a: taken.append(1) or real(*a))
    for tokens in (2, 4, 8, 9):
        for ctx, one_tile in (([64, 20], True), ([64, 65], False)):
            taken.clear()
            _check(ops, heads, kv, size, size, False, 64, ctx, [tokens, 1], one_tile=one_tile)
            assert bool(taken) == (not one_tile or tokens > most)


@pytest.mark.parametrize("heads,kv,size", [(4, 4, 64), (16, 4, 128)])
def test_tiles_of_one_token_cut_from_a_portion(ops, heads, kv, size):
    """Such a token's other keys are written by the kernel in front, so a call that does not say ``alone`` reads nothing of them
    before that kernel has ended; a call that says it with tiles of several tokens is refused."""
    from tinyinfer_b200.kernels.step_lists import row_tiles
    page, ctx, n = 64, 300, 200
    ti = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    positions, table = ti(list(range(ctx - n, ctx))), torch.arange(5, dtype=torch.int32, device=DEV).view(1, 5)
    step = SimpleNamespace(positions=positions, req_of_tok=ti([0] * n), cu_q=ti([0, n]), num_requests=1, max_q_len=n, scratch={})
    proj = torch.randn((n, (heads + 2 * kv) * size), device=DEV)
    rotation = SimpleNamespace(kind="none", rotary_dim=0, inv_freq=None, scale=1.0)
    wq, wk = torch.ones(heads * size, device=DEV), torch.ones(kv * size, device=DEV)
    old = torch.randn((5, kv * page * 2 * size), device=DEV).bfloat16()
    pages, q = old.clone(), torch.empty((n, heads * size), dtype=torch.bfloat16, device=DEV)
    cache = SimpleNamespace(pages=pages, block_table=table, page_size=page, writes=True)
    tiles = ti(row_tiles([n], [ctx - n], 1).tolist())
    part_o, part_ml = torch.empty((n, heads, 2, size), device=DEV), torch.empty((n, heads, 2, 2), device=DEV)
    lib, outs = ops.mixers_tc, []

    def attend(out, tiles, alone):
        return lib.ti_attn_options_tc(
            q.data_ptr(), tiles.data_ptr(), tiles.shape[0], n, positions.data_ptr(), table.data_ptr(), 5, pages.data_ptr(), 5, page,
            heads, kv, size, size, 0, 0, 0, size ** -0.5, 0.0, None, None, None, 0, 0, 2, part_o.data_ptr(), part_ml.data_ptr(), 1,
            alone, out.data_ptr(), ops.status.data_ptr(), torch.cuda.current_stream().cuda_stream)
    for wait in [True] + [False] * 20:
        pages.copy_(old)
        ops.qk_rownorm_rope_store(proj, wq, wk, 1e-6, rotation, step, cache, q, heads, kv, size, size)
        if wait:
            torch.cuda.synchronize()
        outs.append(torch.empty_like(q))
        assert attend(outs[-1], tiles, 0) == 0
    ops.check_status()
    assert all(torch.equal(o, outs[0]) for o in outs[1:])
    assert attend(outs[0], tiles[:n // 2], 1) != 0


@pytest.mark.parametrize("dk,dv,shared,blocks", [(16, 16, 0, 4), (64, 64, 0, 4), (128, 128, 0, 2), (192, 128, 0, 2), (288, 256, 1, 2),
                                                 (576, 512, 1, 1)])
def test_runs_are_counted_by_the_blocks_that_fit(ops, dk, dv, shared, blocks):
    assert ops.mixers_tc.ti_attn_options_tc_run_blocks(dk, dv, shared) == blocks
