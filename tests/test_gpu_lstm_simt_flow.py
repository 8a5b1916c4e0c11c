"""fp32 stacked LSTM whose states carry their own arrival (csrc/lstm_simt_flow.cu): bit for bit the result
of one launch per level."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from fractaltensor_b200 import ops as _ops
    return _ops


def _params(ops, D, H, g):
    u = lambda *s: (torch.rand(*s, device="cuda", generator=g) * 2 - 1) / H ** 0.5
    return ops.lstm_pack_weights(u(D, 4, H, H), u(D, 4, H, H), u(D, 4, H))


@pytest.mark.parametrize("D,L,N,H", [
    (1, 1, 1, 64),      # one step: nothing handed on
    (3, 6, 8, 64),      # a full tile of 8 rows
    (2, 5, 9, 192),     # one sequence in the second tile; a row is not a whole number of warp loads
    (1, 7, 33, 256),    # one layer: narrow tiles spread over the device
    (4, 64, 32, 256),   # tiles of 32, a CTA per tile and layer
    (4, 9, 64, 256),    # layers in groups: weights replaced between sweeps
    (3, 2, 31, 320),    # a row is read in two rounds
    (2, 5, 16, 384),    # the widest state; one input tile beside the weights
    (16, 3, 5, 128),
])
@pytest.mark.parametrize("schedule", [0, 2, 5])  # the automatic choice, the kernel with a counter per cell, this one
def test_same_bits_as_levels(ops, D, L, N, H, schedule):
    g = torch.Generator(device="cuda").manual_seed(D * 100 + N)
    Wp, b = _params(ops, D, H, g)
    x = torch.randn(L, N, H, device="cuda", generator=g)
    ref_h, ref_c = ops.lstm_stacked(x, Wp, b, schedule=1)
    for _ in range(3):  # the fill pattern of a call must not survive into the next
        h, c = ops.lstm_stacked(x, Wp, b, schedule=schedule)
        ops.check_status()
        assert torch.equal(h, ref_h) and torch.equal(c, ref_c)


@pytest.mark.parametrize("D,L,N,H", [
    (3, 24, 36, 192),  # 4 rows: no second cell of a thread
    (4, 40, 48, 128),  # 16: every first cell and no second one
    (2, 20, 49, 256),  # 17: one second cell
])
def test_short_tile_beside_full_ones_of_32_rows(ops, D, L, N, H):
    g = torch.Generator(device="cuda").manual_seed(N)
    Wp, b = _params(ops, D, H, g)
    x = torch.randn(L, N, H, device="cuda", generator=g)
    ref_h, ref_c = ops.lstm_stacked(x, Wp, b, schedule=1)
    h, c = ops.lstm_stacked(x, Wp, b, schedule=5)
    ops.check_status()
    assert torch.equal(h, ref_h) and torch.equal(c, ref_c)


def test_nan_states_are_states(ops):
    """A NaN hidden state is a value like any other (0x7FFFFFFF, not the fill pattern): nothing waits for it."""
    g = torch.Generator(device="cuda").manual_seed(7)
    Wp, b = _params(ops, 2, 128, g)
    x = torch.randn(6, 5, 128, device="cuda", generator=g)
    x[2, 3] = float("nan")
    x.view(torch.int32)[2, 4] = -1  # 0xFFFFFFFF: a NaN with the fill pattern's bits, as an input
    h, _ = ops.lstm_stacked(x, Wp, b, schedule=5)
    ops.check_status()
    assert not torch.isnan(h[:, :, :3]).any() and torch.isnan(h[:, 2:, 3:]).all() and not torch.isnan(h[:, :2]).any()


@pytest.mark.parametrize("D,N,H", [(3, 32, 320), (3, 24, 384), (3, 16, 320), (4, 32, 256), (3, 200, 64)])
def test_automatic_choice_is_the_faster_kernel(ops, D, N, H):
    """Within the 15 % that two timings may differ by; the wrong one is 1.2 to 1.8 times slower at the first two."""
    g = torch.Generator(device="cuda").manual_seed(3)
    Wp, b = _params(ops, D, H, g)
    x = torch.randn(64, N, H, device="cuda", generator=g)

    def us(schedule):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        best = float("inf")
        for _ in range(6):
            e[0].record()
            ops.lstm_stacked(x, Wp, b, schedule=schedule)
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        return best

    assert us(0) <= 1.15 * min(us(2), us(5))


@pytest.mark.parametrize("L,N,I,H", [
    (5, 1, 64, 64),      # two chunks of K in the first step: groups without one
    (4, 32, 64, 128),    # a whole tile
    (6, 33, 320, 192),   # one sequence in the second tile
    (3, 7, 192, 320),
    (4, 40, 512, 256),   # the widest K
])
def test_an_input_of_another_width(ops, L, N, I, H):
    """csrc/lstm_simt_static.cu, the fp32 kernel of models whose input is wider or narrower than the state."""
    g = torch.Generator(device="cuda").manual_seed(I + H)
    u = lambda *s: (torch.rand(*s, device="cuda", generator=g) * 2 - 1) / H ** 0.5
    Wp, b = ops.lstm_pack_weights(u(1, 4, I, H), u(1, 4, H, H), u(1, 4, H))
    x = torch.randn(L, N, I, device="cuda", generator=g)
    ref_h, ref_c = ops.lstm_stacked(x, Wp, b, schedule=1)
    h, c = ops.lstm_stacked(x, Wp, b, schedule=2)
    ops.check_status()
    assert torch.equal(h, ref_h) and torch.equal(c, ref_c)
