"""The native front of the short calls (csrc/host_calls.cpp): it accepts the plain call only and leaves
everything else to the checks in ops.py."""
import pytest
import torch


def test_declines_what_is_not_a_cuda_tensor():
    from fractaltensor_b200._lib import host
    t = torch.zeros(1, 128, 64, dtype=torch.float16)
    q = torch.zeros(1, 1, 256, 128, dtype=torch.float16)
    assert host.b2b_gemm(t, t, t, None, {}) is None
    assert host.b2b_gemm("A", 1, None, None, {}) is None
    assert host.flash_attention(q, q, q, None, 1.0, 0, 0, 0, {}) is None
    assert host.sparse_attention(q, q, q, None, None, 5, 2, 3, 1.0, False, {}) is None


@pytest.mark.gpu
def test_same_errors_and_results_as_the_checked_path():
    from fractaltensor_b200 import ops
    from fractaltensor_b200._lib import FtbError
    A, B, C = (torch.randn(s, device="cuda").half() * 0.1 for s in ((2, 256, 64), (2, 128, 64), (2, 64, 128)))
    ref = ops.b2b_gemm(A, B, C)
    out = torch.empty_like(ref)
    assert ops.b2b_gemm(A, B, C, out) is not None and torch.equal(out, ref)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):  # the caller's current stream, not the default one
        other = ops.b2b_gemm(A, B, C)
    side.synchronize()
    assert torch.equal(other, ref)
    with pytest.raises(ValueError):
        ops.b2b_gemm(A, B, C, out=torch.empty(1, 256, 64, device="cuda", dtype=torch.half))
    with pytest.raises(TypeError):
        ops.b2b_gemm(A, B.float(), C)
    with pytest.raises(ValueError):
        ops.b2b_gemm(A.transpose(1, 2), B, C)
    with pytest.raises(FtbError):
        ops.b2b_gemm(A[:, :100].contiguous(), B, C)
    q = torch.randn(1, 2, 256, 128, device="cuda").half()
    full = ops.flash_attention(q, q, q, scale=1)  # an integer scale takes the checked path
    assert torch.equal(full, ops.flash_attention(q, q, q, scale=1.0)) and torch.equal(full, ops.flash_attention(q, q, q))
    with pytest.raises(ValueError):
        ops.flash_attention(q, q, q, window=4)
    with pytest.raises(FtbError):
        ops.flash_attention(q, q, q, scale=0.0, causal=True)
    with pytest.raises(ValueError):
        ops.sparse_attention(q, q, q, torch.zeros(1, 2, 3, 3, device="cuda", dtype=torch.int32))
    ops.check_status()
