"""The vocabulary projection into rows without gaps (ops.lstm_project_softmax_rows)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from fractaltensor_b200 import ops as _ops
    return _ops


@pytest.mark.parametrize("T,V", [(1, 1), (37, 130), (300, 257), (100, 2000), (64, 9999), (129, 10000), (5, 49151), (9, 256)])
def test_probabilities_without_gaps(ops, T, V):
    """The same numbers as in the padded buffer, for rows that begin on a 16-byte boundary and rows that do not."""
    g = torch.Generator(device="cuda").manual_seed(V)
    P = torch.randn(64, V, device="cuda", generator=g).half()
    h = torch.randn(T, 64, device="cuda", generator=g).half()
    Pt = ops.projection_pack(P)
    rows = ops.lstm_project_softmax_rows(h, Pt, V)
    ops.check_status()
    assert rows.shape == (T, V) and (V % 128 == 0 or rows.is_contiguous())
    assert torch.equal(rows, ops.lstm_project_softmax(h, Pt, V))
    ref = torch.softmax(h.double() @ P.double(), -1)
    # fp32 logits of magnitude up to about 40: 40 * 2^-24 of them, and as much of a probability
    assert (rows.double() - ref).abs().max().item() <= 1e-5
