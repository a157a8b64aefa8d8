"""The table in which a kernel set keeps the answers of its library's size queries, with a library that answers by the
device that is current."""
import sys

from tinyinfer_b200.kernels import CudaOps

cuda_ops = sys.modules[CudaOps.__module__]


class FakeLibrary:
    """Every function exists and returns 1, but the fused feed-forward's sizes fit on device 0 only."""

    def __init__(self):
        self.current, self.asked = 0, 0

    def __getattr__(self, name):
        if name.startswith("__"):
            raise AttributeError(name)

        def function(*args):
            if "ffn_decode_supported" not in name:
                return 1
            self.asked += 1
            return int(self.current == 0)
        setattr(self, name, function)
        return function


def _kernel_set():
    ops = object.__new__(CudaOps)
    ops._bf16 = None
    return ops


def test_kernel_sets_keep_the_answers_of_their_own_device(monkeypatch):
    lib = FakeLibrary()
    monkeypatch.setattr(cuda_ops, "load_library", lambda name: lib)
    sizes = (8, 1024, 3072, 1024, 1024, 3072, 3072, 1024)
    first, second = _kernel_set(), _kernel_set()
    assert [first.bf16.ti_ffn_decode_supported(*sizes) for _ in range(3)] == [1, 1, 1]
    assert lib.asked == 1                                        # answered from the table
    lib.current = 1
    assert second.bf16.ti_ffn_decode_supported(*sizes) == 0      # another device, another answer
    assert first.bf16.ti_ffn_decode_supported(*sizes) == 1
    assert lib.asked == 2
    assert first.bf16 is first.bf16 and first.bf16.ti_gemm_tcgen05_2sm is first.bf16.ti_gemm_tcgen05_2sm
