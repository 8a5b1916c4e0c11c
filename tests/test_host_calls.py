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


def test_calls_of_the_word_program_decline_too():
    from fractaltensor_b200._lib import host
    t = torch.zeros(8, 64, dtype=torch.float16)
    assert host.embedding_gather(t, torch.zeros(3, dtype=torch.int64), None, {}) is None
    assert host.lstm_pack_weights(torch.zeros(1, 4, 64, 64), torch.zeros(1, 4, 64, 64), None) is None
    assert host.lstm_stacked_ragged(t, [8], torch.zeros(1, 256, 128), None, t) is None
    assert host.project_softmax(t, t, {}) is None


def _import_with(prelude):
    """Runs `prelude` and imports the package in a process of its own -> what it printed."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = prelude + """
import warnings
with warnings.catch_warnings(record=True) as seen:
    warnings.simplefilter("always")
    from fractaltensor_b200 import ops
mine = [str(w.message) for w in seen if "_host.so" in str(w.message)]
q = torch.zeros(1, 1, 256, 128, dtype=torch.float16)
for call in (lambda: ops.b2b_gemm(q[0], q[0], q[0]), lambda: ops.flash_attention(q, q, q),
             lambda: ops.sparse_attention(q, q, q, None)):
    try:
        call()
        print("no error")
    except RuntimeError as e:
        assert "CUDA device" in str(e)
print(len(mine), ops.host.__name__)
"""
    return subprocess.run([sys.executable, "-c", code], cwd=root, check=True, capture_output=True, text=True).stdout.split()


def test_the_package_works_without_the_native_front():
    assert _import_with("import torch, sys\nsys.modules['fractaltensor_b200._host'] = None") == ["1", "_NoHost"]


def test_the_native_front_is_not_used_with_another_torch():
    assert _import_with("import torch\ntorch.__version__ = '1.0.0+cpu'") == ["1", "_NoHost"]
    assert _import_with("import torch") == ["0", "fractaltensor_b200._host"]


def test_the_native_front_is_built_again_for_another_torch(monkeypatch):
    import os
    import fractaltensor_b200.build as b
    api = os.path.join(b.HERE, "..", "include", "ftb200.h")
    assert not b._host_is_stale(api)
    monkeypatch.setattr(torch, "__version__", "1.0.0+cpu")
    assert b._host_is_stale(api)


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
