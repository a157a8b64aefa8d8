"""The attention of the 32-bit path against float64 at contexts around the keys that a warp asks for at once, with and
without a window; a row's bits must not depend on how many rows run beside it (which chooses how many keys ahead), nor on
whether the step's lists let blocks take several tokens of a request."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from tinyinfer_b200.kernels import CudaOps
    return CudaOps(DEV)


@pytest.mark.parametrize("heads,kv,d", [(16, 8, 128), (8, 2, 64), (6, 2, 96), (4, 4, 32), (4, 1, 256), (3, 3, 20)])
@pytest.mark.parametrize("window", [None, 11])
def test_rows_alone_and_beside_others(ops, heads, kv, d, window):
    page = 16
    g = torch.Generator(device=DEV).manual_seed(d)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    # every context up to one over eight warps with eight keys each, and a long one
    ctx = [1, 7, 8, 9, 16, 17, 33, 63, 64, 65, 72, 130, 700]
    blocks = [-(-c // page) for c in ctx]
    order = torch.randperm(sum(blocks) + 1, generator=torch.Generator().manual_seed(1)).tolist()
    table = torch.full((len(ctx), max(blocks)), -1, dtype=torch.int32)
    pages = torch.zeros((sum(blocks) + 1, 2, kv, page, d), device=DEV)
    keys, values = [rnd(c, kv, d) for c in ctx], [rnd(c, kv, d) for c in ctx]
    for r, c in enumerate(ctx):
        for b in range(blocks[r]):
            table[r, b] = order.pop()
            n = min(page, c - b * page)
            pages[table[r, b], 0, :, :n] = keys[r][b * page:b * page + n].transpose(0, 1)
            pages[table[r, b], 1, :, :n] = values[r][b * page:b * page + n].transpose(0, 1)
    cache = SimpleNamespace(pages=pages, block_table=table.to(DEV), page_size=page, writes=True)
    # all tokens of all requests: the largest of the three launch shapes of a block per row (the step brings no lists)
    pos, req = [p for c in ctx for p in range(c)], [r for r, c in enumerate(ctx) for _ in range(c)]
    q = rnd(len(pos), heads * d)

    def attend(rows):
        ti = lambda x: torch.tensor([x[i] for i in rows], dtype=torch.int32, device=DEV)
        step = SimpleNamespace(positions=ti(pos), req_of_tok=ti(req), lists={}, scratch={}, max_position=1024, max_ctx_len=700,
                               max_q_len=1, num_tokens=len(rows))
        out = torch.empty((len(rows), heads * d), device=DEV)
        ops.paged_attention(q[rows].contiguous(), step, cache, out, heads, kv, d, window, d ** -0.5)
        return out
    whole = attend(list(range(len(pos))))
    at = 0
    for r, c in enumerate(ctx):
        k, v = (x.double().repeat_interleave(heads // kv, 1) for x in (keys[r], values[r]))
        s = torch.einsum("thd,shd->hts", q[at:at + c].double().view(c, heads, d), k) * d ** -0.5
        i = torch.arange(c, device=DEV)
        dark = i[None] > i[:, None]
        if window:
            dark |= i[None] <= i[:, None] - window
        want = torch.einsum("hts,shd->thd", torch.softmax(s.masked_fill(dark, -torch.inf), -1), v).reshape(c, -1)
        # float32 scores of size d, values near one: some 1e-6
        assert float((whole[at:at + c].double() - want).abs().max()) < 2e-5
        at += c
    last = [sum(ctx[:r + 1]) - 1 for r in range(len(ctx))]
    per_row = heads                                                 # blocks of a row
    for count in (1, ops.num_sms // per_row, ops.num_sms // per_row + 1, 2 * ops.num_sms // per_row):
        for first in range(0, len(last), count):
            rows = last[first:first + count]
            rows = rows + list(range(count - len(rows)))            # filled up to as many rows as the launch shape wants
            assert torch.equal(attend(rows), whole[rows])
        if count * per_row > ops.num_sms:
            rows = last + list(range(100, 100 + max(0, count - len(last))))
            assert torch.equal(attend(rows), whole[rows])
    ops.check_status()


def _step_of(ops, lens, starts, dtype):
    from tinyinfer_b200.engine.batch import build_lists
    ti = lambda x: torch.tensor(np.asarray(x), dtype=torch.int32, device=DEV)
    built = {k: ti(v) for k, v in build_lists(ops.step_lists(dtype), lens, starts).items()}
    return SimpleNamespace(positions=ti([p for n, s in zip(lens, starts) for p in range(s, s + n)]),
                           req_of_tok=ti([r for r, n in enumerate(lens) for _ in range(n)]), lists=built, scratch={},
                           max_position=1024, max_ctx_len=700, max_q_len=max(lens), num_tokens=sum(lens))


# portions on either side of eight tokens a block and of a tile's 64, single tokens in front of, between and behind them; steps
# of too few blocks or too short portions for several tokens a block; single tokens alone
STEPS = [[300], [1, 8, 1, 9, 300, 1, 64, 65, 1], [129, 7, 63, 2, 200] + [1] * 40, [8] * 64, [9] * 70, [2] * 300, [30, 3], [1] * 600,
         [500] + [1] * 500]


@pytest.mark.parametrize("dtype,heads,kv,d", [(torch.float32, 16, 8, 128), (torch.float32, 12, 2, 64), (torch.float32, 20, 4, 20),
                                              (torch.float32, 9, 3, 256), (torch.bfloat16, 10, 5, 20), (torch.bfloat16, 8, 2, 256)])
@pytest.mark.parametrize("lens", STEPS, ids=lambda x: f"{len(x)}x{max(x)}")
def test_several_tokens_a_block(ops, dtype, heads, kv, d, lens):
    page = 16
    starts = [(37 * r) % 150 for r in range(len(lens))]
    g = torch.Generator(device=DEV).manual_seed(len(lens))
    blocks = [-(-(s + n) // page) for n, s in zip(lens, starts)]
    pages = torch.randn((sum(blocks), 2, kv, page, d), generator=g, device=DEV).to(dtype)
    order = torch.randperm(sum(blocks), generator=torch.Generator().manual_seed(1)).tolist()
    table = torch.full((len(lens), max(blocks)), -1, dtype=torch.int32)
    for r, n in enumerate(blocks):
        table[r, :n] = torch.tensor([order.pop() for _ in range(n)])
    cache = SimpleNamespace(pages=pages, block_table=table.to(DEV), page_size=page, writes=True)
    q = torch.randn((sum(lens), heads * d), generator=g, device=DEV).to(dtype)
    outs, launched = [], []
    for window in (1 << 20, None):                                   # a window that hides nothing: always a block per row
        step, before = _step_of(ops, lens, starts, dtype), ops.launches
        out = torch.full_like(q, float("nan"))
        ops.paged_attention(q, step, cache, out, heads, kv, d, window, d ** -0.5)
        outs.append(out)
        launched.append(ops.launches - before)
    assert torch.isfinite(outs[0]).all() and torch.equal(*outs)
    ops.check_status()
    singles = lens.count(1)
    least = 8 if dtype == torch.float32 else max(8, ops._tile_rows[0] // 4)
    shared = (sum(lens) - singles >= least * (len(lens) - singles) > 0 and (sum(lens) - singles) * heads >= 8 * ops.num_sms)
    assert launched == [1, 2 if shared and singles else 1]


def test_a_page_outside_the_pool_is_reported(ops):
    """... by the blocks of several tokens too, and leaves the rows that do not see it alone."""
    from tinyinfer_b200.kernels import KernelError
    page, d = 16, 64
    pages = torch.randn((40, 2, 2, page, d), device=DEV)
    table = torch.arange(40, dtype=torch.int32, device=DEV).view(2, 20)
    q = torch.randn((600, 4 * d), device=DEV)
    outs = []
    for bad in (3, 1 << 20, -5):
        table[1, 3] = 23 if bad == 3 else bad
        step = _step_of(ops, [300, 300], [0, 0], torch.float32)
        out = torch.empty_like(q)
        ops.paged_attention(q, step, SimpleNamespace(pages=pages, block_table=table, page_size=page, writes=True), out, 4, 2, d,
                            None, d ** -0.5)
        outs.append(out)
        if bad == 3:
            ops.check_status()
        else:
            with pytest.raises(KernelError):
                ops.check_status()
            assert torch.equal(out[:348], outs[0][:348])
