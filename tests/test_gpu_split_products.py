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


@pytest.mark.parametrize("m", [1, 4, 6, 40, 130])
@pytest.mark.parametrize("n,k", [(130, 200), (256, 1024), (1024, 520), (40, 4104)])
def test_infinite_weights(ops, m, n, k):
    """An infinite weight gives what a product in float32 gives, also where a row's element has a part that is zero."""
    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.randn((m, k), generator=g, device="cuda")
    a[:, 3] = 1.0                                             # two parts are zero
    a[:, 5] = 0.0
    a[0, 7] = -float("inf")
    w = torch.randn((n, k), generator=g, device="cuda").bfloat16()
    w[1, 3], w[2, 3], w[5, 9], w[6, 5] = float("inf"), -float("inf"), float("inf"), float("inf")
    w[7, 3], w[7, 9], w[8, 2] = float("inf"), -float("inf"), float("nan")
    want = a.double() @ w.double().T
    out = torch.empty((m, n), device="cuda")
    for before in (None, 2.5):
        if before is not None:
            out.fill_(before)
        ops.linear(a, w, out, accumulate=before is not None)
        finite = torch.isfinite(want)
        assert torch.equal(torch.isnan(out), torch.isnan(want))
        assert torch.equal(out[~finite & ~torch.isnan(want)].double(), want[~finite & ~torch.isnan(want)])
        assert bool(((out.double() - want - (before or 0.0)).abs()[finite] <= 1e-4 * k ** 0.5).all())
    assert bool(torch.isinf(want[1:, 1]).all()) and bool(torch.isnan(want[:, 6]).all())
    ops.check_status()


@pytest.mark.parametrize("m", [3, 6, 40])
@pytest.mark.parametrize("exponent", [-90, -105, -110, -115, -120, -126, -133, -140])
def test_small_elements(ops, m, exponent):
    """Elements whose last bits lie below what bfloat16 holds are cut short by less than 2^-133 each, and by nothing from 2^-109
    on; the weights lift the sums out of the range where float32 itself runs short."""
    n, k = 130, 600
    g = torch.Generator(device="cuda").manual_seed(-exponent)
    a = (1.0 + torch.rand((m, k), generator=g, device="cuda")) * 2.0 ** -60 * 2.0 ** (exponent + 60)
    w = (torch.randn((n, k), generator=g, device="cuda") * 2.0 ** 60).bfloat16()
    want = a.double() @ w.double().T
    out = torch.empty((m, n), device="cuda")
    ops.linear(a, w, out)
    cut = 0.0 if exponent >= -109 else 2.0 ** -133 * w.double().abs().sum(1)
    assert bool(((out.double() - want).abs() <= _bound(a, w, k) + cut).all())
    ops.check_status()


@pytest.mark.parametrize("n,k", [(512, 1024), (300, 2048), (130, 4096)])
def test_terms_of_one_sign(ops, n, k):
    """A tensor core cuts its sums off, so terms of one sign leave an error of one sign.  A run's four sums of sixteen terms in
    three parts lose less than four units of 2^-23 of the run, the sums in registers half a unit each and to either side."""
    g = torch.Generator(device="cuda").manual_seed(k)
    a, w = torch.rand((64, k), generator=g, device="cuda") + 0.05, (torch.rand((n, k), generator=g, device="cuda") + 0.05).bfloat16()
    want = a.double() @ w.double().T
    for m in (2, 16, 64):
        out = torch.empty((m, n), device="cuda")
        ops.linear(a[:m], w, out)
        off = (out.double() - want[:m]) / want[:m]
        assert abs(float(off.mean())) < 4 * 2.0 ** -23 and float(off.norm() / off.numel() ** 0.5) < 5 * 2.0 ** -23
    ops.check_status()


@pytest.mark.parametrize("n,k", [(128, 256), (128, 320), (2560, 700), (40, 8192), (1024, 16392), (129, 1030)])
def test_few_rows(ops, n, k):
    """Up to eight rows have a kernel of their own, whose blocks share a tile's K by runs, by chunks or not at all: the bits of a product of
    more rows, next to one another and with rows off a 16-byte boundary, stored and added."""
    g = torch.Generator(device="cuda").manual_seed(n)
    a = torch.randn((70, k), generator=g, device="cuda")
    w = torch.zeros((n, -(-k // 8) * 8), dtype=torch.bfloat16, device="cuda")[:, :k]
    w.copy_(torch.randn((n, k), generator=g, device="cuda"))
    whole = torch.empty((70, n), device="cuda")
    ops.linear(a, w, whole)
    assert bool(((whole.double() - a.double() @ w.double().T).abs() <= _bound(a, w, k)).all())
    for m in (1, 2, 3, 4, 5, 7, 8):
        for first in (0, 9):
            rows = torch.empty(m * (k + 3) + 1, device="cuda")[1:].view(m, k + 3)[:, :k] if first else torch.empty((m, k), device="cuda")
            rows.copy_(a[first:first + m])
            out = torch.full((m, n + 5), 2.0, device="cuda")
            ops.linear(rows, w, out[:, :n])
            assert torch.equal(out[:, :n], whole[first:first + m]) and bool((out[:, n:] == 2.0).all())
            ops.linear(rows, w, out[:, :n], accumulate=True)
            assert torch.equal(out[:, :n], whole[first:first + m] + whole[first:first + m])
    ops.check_status()
