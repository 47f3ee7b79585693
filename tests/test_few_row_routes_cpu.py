"""Which few-row kernel a product reaches, and that products of weights decoded into a scratch just before say so (those kernels ask for weights
ahead of the launch before them). The launches are recorded instead of made."""
import pytest
import torch

from ferrite_b200.ops.cuda_ops import GEMV_MAX_ROWS, CudaOps
from ferrite_b200.ops.qweight import GgufWeight


class Recorder:
    def __init__(self):
        self.calls = []

    def gemv_stream_fits(self, *args):
        return True

    def __getattr__(self, name):
        def call(*args, **kw):
            self.calls.append((name, args, kw))
            return 0
        return call


def recording_ops():
    ops = CudaOps.__new__(CudaOps)
    ops.__dict__.update(C=Recorder(), dtype=torch.bfloat16, device=torch.device("cpu"), empty=torch.empty, launches=0, sm_count=148, _scratch={},
                        mma_gemv_rows=(2, 32), force_gemv_chunks=False, _ws=torch.empty(1 << 22), _stream_bytes=16, _counters=torch.zeros(1, dtype=torch.int32),
                        status_word=torch.zeros(1, dtype=torch.int32))
    return ops


# wide rows (no GEMV on the blocks), small and large matrices: the three few-row kernels
@pytest.mark.parametrize("rows,n,kernel", [(1, 64, "gemv"), (2, 64, "gemv_mma"), (8, 64, "gemv_mma"), (32, 64, "gemv_mma"), (2, 1300, "gemv_stream"),
                                           (9, 1300, "gemv_stream"), (32, 1300, "gemv_stream")])
def test_scratch_copies_are_told_apart(rows, n, kernel):
    ops, K = recording_ops(), 6656
    x = torch.zeros(rows, K, dtype=torch.bfloat16)
    assert rows > GEMV_MAX_ROWS or K * 32 > 200 * 1024
    ops.linear(x, GgufWeight(torch.zeros(1, dtype=torch.uint8), 8, n, K))
    assert [c[0] for c in ops.C.calls] == ["gguf_dequant", kernel]
    assert ops.C.calls[1][1][-1] is True
    ops.C.calls.clear()
    ops.linear(x, torch.zeros(n, K, dtype=torch.bfloat16))
    assert ops.C.calls[0][0] == kernel and ops.C.calls[0][1][-1] is False
