"""Products of float32 rows with bfloat16 weights on the tensor cores: sizes around a run, a chunk, a tile of weights and of
tokens, and on either side of every way a tile's K is cut.  A run of 64 terms is four sums of sixteen, cut off to 23 bits in
three parts; runs, chunks and the total are rounded sums, so an element lies within (8 + runs + chunks + 2) units of 2^-23 of
its terms' magnitude, and the whole within 2e-7 of the norm.  A row's bits must not depend on the rows beside it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from tinyinfer_b200.kernels import CudaOps
    ops = CudaOps("cuda:0")
    ops.split_from = 0
    return ops


def _bound(a, w, k):
    return (8 + -(-k // 64) + -(-k // 512) + 2) * 2.0 ** -23 * (a.double().abs() @ w.double().abs().T)


@pytest.mark.parametrize("n,k", [(1, 8), (127, 64), (128, 65), (129, 72), (200, 320), (200, 321), (130, 512), (130, 520),
                                 (1024, 1024), (300, 1025), (6144, 1024), (257, 1536), (40, 4104), (20000, 128)])
def test_rows_of_every_number(ops, n, k):
    g = torch.Generator(device="cuda").manual_seed(n + k)
    a = torch.randn((200, k), generator=g, device="cuda") * torch.randn((200, 1), generator=g, device="cuda").exp()
    w = torch.zeros((n, -(-k // 8) * 8), dtype=torch.bfloat16, device="cuda")[:, :k]
    w.copy_(torch.randn((n, k), generator=g, device="cuda"))
    want = a.double() @ w.double().T
    whole = torch.empty((200, n), device="cuda")
    ops.linear(a, w, whole)
    assert bool(((whole.double() - want).abs() <= _bound(a, w, k)).all())
    assert float((whole.double() - want).norm() / want.norm()) < 2e-7
    for m in (1, 2, 3, 4, 5, 15, 16, 17, 63, 64, 65, 129):
        out = torch.full((m, n), 3.0, device="cuda")
        ops.linear(a[:m], w, out)
        assert torch.equal(out, whole[:m]), m
        ops.linear(a[:m], w, out, accumulate=True)
        assert torch.equal(out, whole[:m] + whole[:m]), m
    shifted = torch.empty(9 * (k + 1) + 1, device="cuda")[1:].view(9, k + 1)[:, :k]      # rows off a 16-byte boundary
    shifted.copy_(a[:9])
    out = torch.empty((9, n + 3), device="cuda")[:, 1:n + 1]
    ops.linear(shifted, w, out)
    assert torch.equal(out, whole[:9])
    ops.check_status()


def test_numbers_at_the_ends_of_their_range(ops):
    """Infinite and NaN elements stay in their rows; the largest numbers do not overflow in parts; zeros are exact."""
    k = 192
    a = torch.randn((6, k), device="cuda")
    w = torch.randn((130, k), device="cuda").bfloat16()
    w[3] = 0.0
    a[1, 7], a[2, 100], a[3, 50] = float("inf"), float("nan"), -float("inf")
    a[4] = 0.0
    a[4, 9] = 3.4028234e38
    w[:, 9] = 0.5
    out = torch.empty((6, 130), device="cuda")
    ops.linear(a, w, out)
    assert torch.isfinite(out[0]).all() and torch.isfinite(out[5]).all()
    sign = w[:, 7].float().sign()
    live = sign != 0
    assert torch.equal(out[1][live], sign[live] * float("inf")) and torch.isnan(out[1][~live]).all()
    assert torch.isnan(out[2]).all()
    assert torch.equal(out[3][w[:, 50] != 0], -w[:, 50].float().sign()[w[:, 50] != 0] * float("inf"))
    assert torch.equal(out[4], torch.full((130,), 0.5 * 3.4028234e38, device="cuda"))
    ops.check_status()
