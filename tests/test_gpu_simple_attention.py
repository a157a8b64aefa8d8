"""The attention of the 32-bit path against float64 at contexts around the keys that a warp asks for at once, with and
without a window; a row's bits must not depend on how many rows run beside it (which chooses how many keys ahead)."""
from types import SimpleNamespace

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
    # all tokens of all requests: the largest of the three launch shapes
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
