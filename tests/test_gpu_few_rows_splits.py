"""The split-K tcgen05 product of few rows where its rule changes: few tiles cut into two to six splits, whole tiles, and
two splits of more units than the grid holds."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from tinyinfer_b200.kernels import CudaOps
    return CudaOps("cuda:0")


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
