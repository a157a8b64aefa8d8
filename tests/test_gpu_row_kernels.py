"""The row kernels of decode steps in both of their forms (four elements at a time, element by element) against float64, at
the sizes where the forms meet: heads that are no multiple of four, rows that fill or just miss a thread's units, one token
and several, columns and inputs of the products per head beside their tiles.  float32 results are held to 2e-6 of the row's
largest value (a few roundings of 2^-24, and 2^-22 of the sine), bfloat16 ones to one rounding (2^-8) more."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64
PAGE = 16


@pytest.fixture(scope="module")
def ops():
    from tinyinfer_b200.kernels import cuda_ops
    return cuda_ops(DEV)


def _rand(shape, seed, dtype=torch.float32):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(DEV).to(dtype)


def _near(got, want, what):
    tol = 2e-6 + (2.0 ** -8 if got.dtype == torch.bfloat16 else 0.0)
    want = want.to(F64)
    bound = tol * (want.abs() if got.dtype == torch.bfloat16 else 0.0) + 2e-6 * want.abs().amax(-1, keepdim=True)
    assert ((got.to(F64) - want).abs() <= bound).all(), (what, (got.to(F64) - want).abs().max().item())


def _step(lengths, starts):
    ti = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    pos = [p for n, s in zip(lengths, starts) for p in range(s, s + n)]
    cu = [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    return SimpleNamespace(positions=ti(pos), req_of_tok=ti([r for r, n in enumerate(lengths) for _ in range(n)]), cu_q=ti(cu),
                           num_requests=len(lengths), max_q_len=max(lengths), scratch={})


def _cache(step, per_token, dtype, writes=True):
    blocks = int(step.positions.max()) // PAGE + 1
    n = step.num_requests
    order = torch.randperm(n * blocks, generator=torch.Generator().manual_seed(1)).to(torch.int32)
    return SimpleNamespace(pages=torch.zeros((n * blocks, per_token * PAGE), dtype=dtype, device=DEV),
                           block_table=order.view(n, blocks).to(DEV), page_size=PAGE, writes=writes)


def _stored(cache, step, base, head, size, per_page):
    """Element rows of one head as the pages hold them: ``[T, size]``; ``base``: where that kind starts in a page."""
    pos, req = step.positions.long(), step.req_of_tok.long()
    page = cache.block_table.long()[req, pos // PAGE]
    at = base + (head * PAGE + pos % PAGE) * size
    return cache.pages.view(-1, per_page)[page[:, None], at[:, None] + torch.arange(size, device=DEV)]


def _turn(x, pos, freq, halves, mag=1.0):
    """x [T, n] float64, first 2 * len(freq) elements turned."""
    half = freq.numel()
    ang = (pos.to(torch.float32)[:, None] * freq[None]).to(F64)          # the angle is a float32 product
    c, s = torch.cos(ang) * mag, torch.sin(ang) * mag
    y = x.clone()
    a, b = (x[:, :half], x[:, half:2 * half]) if halves else (x[:, 0:2 * half:2], x[:, 1:2 * half:2])
    ya, yb = a * c - b * s, b * c + a * s
    if halves:
        y[:, :half], y[:, half:2 * half] = ya, yb
    else:
        y[:, 0:2 * half:2], y[:, 1:2 * half:2] = ya, yb
    return y


def _freq(rot):
    return 10000.0 ** (-torch.arange(rot // 2, device=DEV, dtype=torch.float32) * 2 / max(rot, 1))


# heads, kv heads, dk, dv, rotated: units of four and one that misses them; 512 units, 516; 2,048 units and 2,056 (the general form)
SHAPES = [(4, 2, 64, 64, 64), (2, 1, 20, 12, 8), (3, 1, 10, 6, 6), (2, 2, 24, 20, 6), (31, 1, 64, 64, 32), (42, 1, 48, 16, 48),
          (60, 4, 128, 32, 128), (253, 4, 32, 8, 32), (16, 4, 128, 128, 0)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lengths,starts", [([1], [70]), ([1, 1, 1], [0, 15, 40]), ([5, 1, 9], [3, 0, 100])])
@pytest.mark.parametrize("heads,kv,dk,dv,rot", SHAPES)
def test_rows_of_heads(ops, heads, kv, dk, dv, rot, lengths, starts, dtype):
    step = _step(lengths, starts)
    t, nq, nk, nv = sum(lengths), heads * dk, kv * dk, kv * dv
    proj = _rand((t, nq + nk + nv + 4), 3)
    x, pos, freq = proj.to(F64), step.positions, _freq(rot)
    wq, wk = _rand((nq,), 4), _rand((nk,), 5)
    per_page = (dk + dv) * kv * PAGE

    def check(q, cache, norm, halves, mag, values, head_norm=False):
        for part, n, count, w in (("q", nq, heads, wq), ("k", nk, kv, wk)):
            row = x[:, :nq] if part == "q" else x[:, nq:nq + nk]
            if norm:
                row = row / torch.sqrt((row * row).mean(-1, keepdim=True) + 1e-6) * w.to(F64)
            for h in range(count):
                head = row[:, h * dk:(h + 1) * dk]
                if head_norm:
                    head = head / torch.sqrt((head * head).mean(-1, keepdim=True) + 1e-6) * (wq if part == "q" else wk)[:dk].to(F64)
                want = _turn(head, pos, freq, halves, mag)
                got = q.view(t, heads, dk)[:, h] if part == "q" else _stored(cache, step, 0, h, dk, per_page)
                _near(got, want, (part, h))
        for h in range(kv):
            _near(_stored(cache, step, kv * PAGE * dk, h, dv, per_page), values[:, h * dv:(h + 1) * dv], ("v", h))

    v = x[:, nq + nk:nq + nk + nv]
    q = torch.empty((t, nq), dtype=dtype, device=DEV)
    rotation = SimpleNamespace(kind="interleaved" if rot else "none", rotary_dim=rot, inv_freq=freq, scale=1.0)
    for per_head in (False, True):
        cache = _cache(step, kv * (dk + dv), dtype)
        ops.qk_rownorm_rope_store(proj, wq[:dk].contiguous() if per_head else wq, wk[:dk].contiguous() if per_head else wk, 1e-6,
                                  rotation, step, cache, q, heads, kv, dk, dv, per_head=per_head)
        check(q, cache, not per_head, False, 1.0, v, head_norm=per_head)
    first = _rand((t, nv), 6)
    mixed = 0.75 * v + 0.25 * first.to(F64)
    halves = SimpleNamespace(kind="neox" if rot else "none", rotary_dim=rot, inv_freq=freq, scale=1.25)
    cache = _cache(step, kv * (dk + dv), dtype)
    ops.qkv_turn_store(proj, halves, None, step, cache, q, heads, kv, dk, dv, value_mix=(first, 0.25))
    check(q, cache, False, True, 1.25, mixed)
    ops.check_status()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lengths,starts", [([1], [33]), ([3, 1], [15, 0])])
@pytest.mark.parametrize("heads,dk,dr,rank", [(16, 64, 32, 256), (3, 6, 4, 10), (2, 8, 0, 1028), (5, 20, 12, 64)])
def test_latent_rows(ops, heads, dk, dr, rank, lengths, starts, dtype):
    step = _step(lengths, starts)
    t, row = sum(lengths), rank + dr
    proj = _rand((t, heads * (dk + dr) + row), 7)
    w, freq = _rand((rank,), 8), _freq(dr)
    cache = _cache(step, row, dtype)
    plain = torch.empty((t, heads, dk), dtype=dtype, device=DEV)
    full = torch.zeros((t, heads, row), dtype=dtype, device=DEV)
    rotation = SimpleNamespace(kind="interleaved" if dr else "none", rotary_dim=dr, inv_freq=freq, scale=1.0)
    ops.latent_prepare(proj, w, 1e-5, rotation, step, cache, plain.view(t, -1), full, heads, dk, dr, rank)
    x = proj.to(F64)
    for h in range(heads):
        head = x[:, h * (dk + dr):(h + 1) * (dk + dr)]
        _near(plain[:, h], head[:, :dk], ("plain", h))
        if dr:
            _near(full[:, h, rank:], _turn(head[:, dk:], step.positions, freq, False), ("turned", h))
    lat = x[:, heads * (dk + dr):]
    want = lat[:, :rank] / torch.sqrt((lat[:, :rank] ** 2).mean(-1, keepdim=True) + 1e-5) * w.to(F64)
    got = _stored(cache, step, 0, 0, row, row * PAGE)
    _near(got[:, :rank], want, "latent")
    if dr:
        _near(got[:, rank:], _turn(lat[:, rank:], step.positions, freq, False), "key part")
    ops.check_status()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width", [4, 1022, 1024, 1028, 2048])
@pytest.mark.parametrize("n_mix", [5, 3])
def test_token_shift(ops, n_mix, width, dtype):
    step = _step([1, 4, 2], [9, 0, 5])
    h, mu = _rand((7, width), 9, dtype), _rand((n_mix, width), 10)
    state = SimpleNamespace(state=_rand((4, 8 + width), 11), slots=torch.tensor([2, 0, 3], dtype=torch.int32, device=DEV))
    out = torch.empty((n_mix, 7, width), dtype=dtype, device=DEV)
    ops.token_shift_mix(h, mu, step, state, 8, out)
    x = h.to(F64)
    before = torch.cat([x[:1], x[:-1]])
    for i, r in ((0, 2), (1, 0), (5, 3)):
        before[i] = state.state[r, 8:].to(F64)
    for s in range(n_mix):
        _near(out[s], x + (before - x) * mu[s].to(F64), s)


@pytest.mark.parametrize("n", [4 * 1024, 1023, 1])
def test_rows_through_an_activation(ops, n):
    x = _rand((1, n), 12) * 3.0
    for dtype in (torch.float32, torch.bfloat16):
        out = torch.empty((1, n), dtype=dtype, device=DEV)
        z = x.to(F64)
        ops.xielu_rows(x, 0.8, 1.3, out)
        _near(out, torch.where(z > 0, 0.8 * z * z + 0.5 * z, 1.3 * (torch.expm1(z) - z) + 0.5 * z), "xielu")
        ops.tanh_rows(x, out)
        _near(out, torch.tanh(z), "tanh")


@pytest.mark.parametrize("t", [1, 4, 5, 8, 9, 16, 17, 64])
@pytest.mark.parametrize("n_in,n_out", [(128, 512), (512, 128), (129, 36), (600, 33), (8, 4), (3, 2)])
def test_products_per_head_of_few_tokens(ops, t, n_in, n_out):
    """A row's bits depend on the row alone; sums of n_in float32 terms in front of one bfloat16 rounding."""
    heads = 3
    x, w = _rand((t, heads, n_in), 13, torch.bfloat16), _rand((heads, n_in, n_out), 14, torch.bfloat16)
    out = torch.empty((t, heads, n_out), dtype=torch.bfloat16, device=DEV)
    ops.head_project(x, w, out)
    want = torch.einsum("thk,hkn->thn", x.to(F64), w.to(F64))
    terms = torch.einsum("thk,hkn->thn", x.to(F64).abs(), w.to(F64).abs())
    assert ((out.to(F64) - want).abs() <= 2.0 ** -8 * want.abs() + n_in * 2.0 ** -24 * terms).all()
    alone = torch.empty((1, heads, n_out), dtype=torch.bfloat16, device=DEV)
    ops.head_project(x[t - 1:], w, alone)
    assert torch.equal(alone[0], out[t - 1])


@pytest.mark.parametrize("hidden", [4, 1022, 1024, 1028, 5120])
def test_embedding_rows(ops, hidden):
    tokens = torch.tensor([3, 0, 6, 3], dtype=torch.int32, device=DEV)
    for dtype in (torch.float32, torch.bfloat16):
        table = _rand((7, hidden), 15, dtype)
        out = torch.empty((4, hidden), device=DEV)
        ops.embed(table, tokens, out)
        assert torch.equal(out, table[tokens.long()].float())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,kv,dk", [(16, 4, 128), (31, 1, 64), (32, 1, 64), (60, 4, 64), (61, 4, 64), (60, 4, 128)])
def test_a_row_of_heads_does_not_depend_on_the_rows_beside_it(ops, heads, kv, dk, dtype):
    """300 rows and the same rows in runs of 1, 7 and 255, on either side of every number of units and tokens that chooses a
    launch shape (512 and 1,024 units, 256 tokens)."""
    t, nq, nk = 300, heads * dk, kv * dk
    proj, wq, wk, freq = _rand((t, nq + 2 * nk), 1), _rand((nq,), 2), _rand((nk,), 3), _freq(dk)
    rotation = SimpleNamespace(kind="interleaved", rotary_dim=dk, inv_freq=freq, scale=1.0)

    def rows(first, n):
        step = _step([n], [first])
        cache = _cache(step, kv * 2 * dk, dtype)
        q = torch.empty((n, nq), dtype=dtype, device=DEV)
        ops.qk_rownorm_rope_store(proj[first:first + n], wq, wk, 1e-6, rotation, step, cache, q, heads, kv, dk, dk)
        per_page = 2 * dk * kv * PAGE
        kept = [_stored(cache, step, base * kv * PAGE * dk, h, dk, per_page) for base in (0, 1) for h in range(kv)]
        return torch.cat([q] + kept, 1)
    whole = rows(0, t)
    for run in (1, 7, 255):
        for first in (0, 20, 45):
            assert torch.equal(rows(first, run), whole[first:first + run]), (run, first)
