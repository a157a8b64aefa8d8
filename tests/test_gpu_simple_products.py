"""The float32 products at the edges of their kernels: rows around the streaming kernel's groups and limit, inner sizes
around a segment, a span and a round, columns around a warp's and a tile's, rows that cannot be read 16 bytes at a
time.  Every element must lie within the rounding of its sums, and a row's bits must not depend on how many rows
run beside it, nor on the alignment of the operands (which chooses the kernel)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SEG = 256


@pytest.fixture(scope="module")
def ops():
    from tinyinfer_b200.kernels import CudaOps
    return CudaOps("cuda:0")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,k", [(8, 8), (33, 248), (70, 256), (2049, 264), (1024, 1024), (40, 1032), (17, 2048), (24, 4104),
                                 (65, 36), (9, 1001)])
def test_float32_products(ops, dtype, n, k):
    g = torch.Generator(device="cuda").manual_seed(n * 7 + k)
    rows = torch.randn((130, k), generator=g, device="cuda")
    w = torch.randn((n, k), generator=g, device="cuda").to(dtype)
    want = rows.double() @ w.double().T
    # a segment's running sum of at most SEG terms, then at most k / SEG sums: each rounds by half a unit
    bound = (min(k, SEG) + k // SEG + 2) * 2.0 ** -24 * (rows.double().abs() @ w.double().abs().T)
    whole = torch.empty((130, n), device="cuda")
    ops.linear(rows, w, whole)
    assert bool(((whole.double() - want).abs() <= bound).all())
    for m in (1, 2, 3, 4, 5, 8, 9, 32, 33, 64, 65):
        out = torch.full((m, n), 3.0, device="cuda")
        ops.linear(rows[:m], w, out)
        assert torch.equal(out, whole[:m]), m
        ops.linear(rows[:m], w, out, accumulate=True)
        assert torch.equal(out, whole[:m] + whole[:m]), m
    # operands one element off a 16-byte boundary take the tiles
    shifted = torch.empty(9 * (k + 1) + 1, device="cuda")[1:].view(9, k + 1)[:, :k]
    shifted.copy_(rows[:9])
    out = torch.empty((9, n), device="cuda")
    ops.linear(shifted, w, out)
    assert torch.equal(out, whole[:9])
