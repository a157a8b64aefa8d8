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


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,k", [(8, 8), (128, 64), (256, 256), (5120, 5120), (32768, 8)])
def test_few_rows_cost_no_more_than_a_tile(ops, dtype, n, k):
    """Up to 32 rows choose between two kernels: none may take longer than 33 rows, which take the tiles (half as much
    again is left to the clock)."""
    w = torch.randn((n, k), device="cuda").to(dtype)

    def microseconds(m):
        rows, out = torch.randn((m, k), device="cuda"), torch.empty((m, n), device="cuda")
        side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.stream(side):
            ops.linear(rows, w, out)
        side.synchronize()
        with torch.cuda.graph(graph, stream=side):
            for _ in range(20):
                ops.linear(rows, w, out)
        times = []
        for _ in range(5):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            with torch.cuda.stream(side):
                start.record()
                graph.replay()
                end.record()
            end.synchronize()
            times.append(start.elapsed_time(end) * 50)
        return min(times)
    most = 1.5 * microseconds(33)
    for m in (1, 8, 17, 32):
        assert microseconds(m) <= most, m


@pytest.mark.parametrize("k", [200, 256, 300, 512, 513])
def test_many_tiles_of_few_segments(ops, k):
    """One, two and four groups of warps per tile give the same bits: row counts on either side of the limits."""
    g = torch.Generator(device="cuda").manual_seed(k)
    rows, w = (torch.randn((s, k), generator=g, device="cuda") for s in (1300, 1000))
    want = rows.double() @ w.double().T
    bound = (min(k, SEG) + k // SEG + 2) * 2.0 ** -24 * (rows.double().abs() @ w.double().abs().T)
    whole = torch.empty((1300, 1000), device="cuda")
    ops.linear(rows, w, whole)
    assert bool(((whole.double() - want).abs() <= bound).all())
    for m in (33, 500, 640, 1100):            # 16, 128, 160 and 288 tiles; the whole product has 336
        out = torch.empty((m, 1000), device="cuda")
        ops.linear(rows[:m], w, out)
        assert torch.equal(out, whole[:m]), m
