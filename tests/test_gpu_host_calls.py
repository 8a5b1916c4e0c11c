"""The native front of the short calls on a device: what a caller and the other threads of the program see."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _b2b(batch=1, M=128):
    g = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).half() * 0.1
    return r(batch, M, 64), r(batch, 128, 64), r(batch, 64, 128)


def test_no_room_for_the_result_is_torch_s_own_error():
    from fractaltensor_b200 import ops
    z = lambda *s: torch.zeros(*s, device="cuda", dtype=torch.half)  # (no temporaries: nothing is left to reuse)
    torch.cuda.empty_cache()
    A, B, C, q = z(4, 1 << 17, 64), z(4, 128, 64), z(4, 64, 128), z(1, 8, 32768, 128)  # results of 64 MB
    ops.b2b_gemm(*_b2b())  # the workspace exists: the native front takes the calls
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.set_per_process_memory_fraction(1e-6)
    try:
        for call in (lambda: ops.b2b_gemm(A, B, C), lambda: ops.flash_attention(q, q, q, causal=True),
                     lambda: ops.sparse_attention(q, q, q, None)):
            with pytest.raises(torch.OutOfMemoryError):
                call()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert ops.b2b_gemm(A, B, C).shape == (4, 1 << 17, 64)
