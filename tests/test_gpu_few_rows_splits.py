"""The split-K tcgen05 product of few rows where its rule changes: few tiles cut into up to nine splits, whole tiles, and
splits of more units than the grid holds."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from tinyinfer_b200.kernels import CudaOps
    return CudaOps("cuda:0")


def _splits(ops, m, n, k):
    """In how many splits the product cuts K, from the size of the workspace it asks for."""
    floats, tickets = ctypes.c_longlong(-1), ctypes.c_int(-1)
    ops.bf16.ti_gemm_tcgen05_few_scratch(m, n, k, ctypes.byref(floats), ctypes.byref(tickets))
    tiles = -(-n // 128)
    assert tickets.value == tiles
    rows = 16 if m <= 16 else 32 if m <= 32 else 64
    return max(1, floats.value // (tiles * rows * 128))


# splits on 148 SMs: fewer units than SMs, one to two units an SM, a round and a few units, whole tiles
SPLITS = {(2048, 12288): 9, (4096, 12288): 8, (5120, 8192): 6, (10240, 5120): 3, (12288, 2048): 3, (15104, 2048): 2,
          (15232, 2048): 2, (18944, 1024): 1, (38016, 2048): 1, (38016, 17408): 4}


@pytest.mark.parametrize("n,k", list(SPLITS))
def test_the_rule_cuts_as_measured(ops, n, k):
    if ops.num_sms != 148:
        pytest.skip("the expected splits are for 148 SMs")
    for m in (1, 16, 17, 64):
        assert _splits(ops, m, n, k) == SPLITS[n, k]


@pytest.mark.parametrize("n,k", [(4096, 12288), (15104, 2048), (38016, 2048)])
def test_epilogues_behind_splits(ops, n, k):
    """SwiGLU and a gated sum behind eight splits, two, and whole tiles."""
    from tinyinfer_b200.parts.base import GatedSum
    g = torch.Generator(device="cuda").manual_seed(n)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    w = rnd(n, k).bfloat16()
    rows = (rnd(64, k) * k ** -0.5).bfloat16()
    gate, up = w[:n // 2], w[n // 2:]
    packed = ops.pack_gate_up(gate.contiguous(), up.contiguous())
    gates, bias, x = rnd(64, n), rnd(n), rnd(64, n)
    # float32 sums of values near one: errors of some 1e-6, far below half a unit of bfloat16
    prod = rows.double() @ w.double().T
    glu = torch.nn.functional.silu(prod[:, :n // 2]) * prod[:, n // 2:]
    sums = x.double() + 0.7 * torch.sigmoid(gates.double() + bias.double()) * prod
    for m in (1, 16, 33, 64):
        out = torch.empty((m, n // 2), dtype=torch.bfloat16, device="cuda")
        assert ops._few_tc(rows[:m], packed, None, out, 2)
        assert bool(((out.double() - glu[:m]).abs() <= glu[:m].abs() * 2.0 ** -8 + 1e-5).all())
        y = x[:m].clone()
        ops.linear(rows[:m], w, GatedSum(y, gates[:m], bias, 0.7), accumulate=True)
        assert bool(((y.double() - sums[:m]).abs() <= 1e-5 * (1 + sums[:m].abs())).all())
    ops.check_status()


@pytest.mark.parametrize("n,k", [(4096, 12288), (5120, 8192), (10240, 5120), (15104, 2048), (15232, 2048), (38016, 17408)])
def test_splits_of_few_rows(ops, n, k):
    g = torch.Generator(device="cuda").manual_seed(n)
    w = torch.randn((n, k), generator=g, device="cuda", dtype=torch.bfloat16)
    rows = torch.randn((64, k), generator=g, device="cuda").bfloat16()
    base = torch.randn((64, n), generator=g, device="cuda")
    # a sample of columns, the first and the last tile among them
    cols = torch.cat([torch.arange(0, 128), torch.randint(0, n, (256,), generator=torch.Generator().manual_seed(1)),
                      torch.arange(n - 128, n)]).to("cuda")
    a, b = rows.double(), w[cols].double()
    want = a @ b.T
    # float32 sums in an order of the kernel's own: k / 16 steps that each round a running sum of at most some |a| |b| / k^.5
    bound = 16 * 2.0 ** -24 * (a.norm(dim=1)[:, None] * b.norm(dim=1)[None]) + 1e-6
    full = torch.empty((64, n), device="cuda")
    ops.linear(rows, w, full)
    for m in (1, 16, 17, 33, 64):
        out = torch.full((m, n), 5.0, device="cuda")
        assert ops._few_tc(rows[:m], w, out, None, 0)
        assert torch.equal(out, full[:m]), "a row's bits depend on the rows beside it"
        added = base[:m].clone()
        ops.linear(rows[:m], w, added, accumulate=True)
        assert bool(((added[:, cols].double() - (base[:m][:, cols].double() + want[:m])).abs()
                     <= bound[:m] + 2.0 ** -23 * (base[:m][:, cols].abs() + want[:m].abs())).all())
    assert bool(((full[:, cols].double() - want).abs() <= bound).all())
    ops.check_status()
