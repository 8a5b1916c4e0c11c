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


@pytest.mark.parametrize("rows,width", [(3, 2), (40, 131), (9, 1028), (30, 5001), (5, 20001), (2, 60003), (2, 60004)])
def test_softmax_of_rows_that_begin_anywhere(ops, rows, width):
    """Rows of x, of y or of both off the 16-byte boundary; both sizes of CTA, and rows longer than the on-chip cache."""
    g = torch.Generator(device="cuda").manual_seed(width)
    x = torch.randn(rows, width, device="cuda", generator=g) * 3
    ref = torch.softmax(x.double(), -1)
    for at_x, at_y in ((0, 0), (0, 1), (3, 0), (1, 2)):
        bx, by = (torch.full((rows * width + 4,), 7.0, device="cuda") for _ in range(2))
        xs, ys = bx[at_x:at_x + rows * width].view(rows, width), by[at_y:at_y + rows * width].view(rows, width)
        xs.copy_(x)
        ops.online_softmax(xs, ys)
        # fp32 sums of up to 60004 terms and an exponential of relative error 2^-22 or so
        assert ((ys.double() - ref).abs() / ref).max().item() <= 1e-4
        assert by[:at_y].eq(7).all() and by[at_y + rows * width:].eq(7).all()
