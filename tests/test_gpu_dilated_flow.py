"""Dilated LSTM without clusters (csrc/rnn_cluster.cu): layers of dilation 1 on slices of 16, 32 or 48 sequences, and of
dilation 2 where they fit, hand their state on through the output array, the others are on slices of 64 or 128; bit for bit the
result of one launch per level."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from fractaltensor_b200 import ops as _ops
    return _ops


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("L,N,H,dils", [
    (9, 17, 256, [1]),                       # 16 wide, one sequence in the second slice
    (12, 128, 256, [1, 2, 4]),               # 16 beside 64
    (13, 256, 256, [1, 2, 4]),               # 32 beside 64
    (40, 256, 256, [1, 2, 4, 8, 16, 32]),    # 48 beside 64 and 128: slices that straddle those below
    (11, 200, 256, [4, 1, 2, 8, 3, 5]),      # the same with the narrow layer on top of a wide one
    (10, 300, 128, [2, 1, 1, 4]),            # two narrow layers
    (7, 90, 64, [1, 2]),
])
def test_same_bits_as_levels(ops, dt, L, N, H, dils):
    _against_levels(ops, dt, L, N, H, dils, 5)


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("L,N,H,dils", [
    (9, 33, 128, [1]),              # clusters of 4 CTAs, here and below; then of 2
    (20, 64, 128, [1, 2, 4]),
    (20, 64, 64, [1, 1, 2]),
    (7, 5, 64, [1, 3]),
    (12, 128, 256, [1, 2, 4]),      # 8 CTAs: state pieces for eight peers
    (11, 256, 256, [1, 2, 4, 8]),   # slices of 64 below slices of 128
    (9, 256, 256, [4, 1, 2]),       # slices of 128 below slices of 64
    (6, 300, 128, [4, 1, 2]),       # partly filled slices
])
@pytest.mark.parametrize("schedule", [4, 0])
def test_clusters_same_bits_as_levels(ops, dt, L, N, H, dils, schedule):
    """One thread-block cluster per layer and slice (schedule 4); the automatic choice takes it for short sequences of 64 units."""
    _against_levels(ops, dt, L, N, H, dils, schedule)


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_nan_states_are_states(ops, dt):
    """A NaN hidden state of a layer with dilation 1 is not the fill pattern: nothing waits for it."""
    N, H, dils = 20, 64, [1, 2, 1]
    g = torch.Generator(device="cuda").manual_seed(7)
    u = lambda *s: ((torch.rand(*s, device="cuda", generator=g) * 2 - 1) / H ** 0.5).to(dt)
    Wp, b = ops.lstm_pack_weights(u(3, 4, H, H), u(3, 4, H, H), u(3, 4, H))
    x = torch.randn(6, N, H, device="cuda", generator=g).to(dt)
    x[2, 3] = float("nan")
    x.view(torch.int16)[2, 4] = -1  # 0xFFFF: a NaN with the fill pattern's bits, as an input
    ref, _ = ops.lstm_dilated(x, Wp, dils, b, schedule=1)
    h, _ = ops.lstm_dilated(x, Wp, dils, b, schedule=5)
    ops.check_status()
    assert torch.isnan(h[:, 2:, 3:5]).any() and torch.equal(torch.isnan(h), torch.isnan(ref))
    assert torch.equal(torch.nan_to_num(h), torch.nan_to_num(ref))


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("L,N,H,dils", [
    (1, 5, 128, [1, 2]),             # one step: half of the second layer's columns have none
    (2, 17, 64, [2, 1]),             # the folded layer reads the input
    (7, 9, 256, [1, 2, 2]),          # an odd number of steps; folded on folded, slices that straddle two time steps
    (23, 33, 256, [1, 2, 4, 2, 1]),  # beside cells of dilation 4, above and below
    (30, 100, 128, [1, 2, 4, 8]),
    (12, 256, 128, [1, 2]),
])
def test_layers_of_dilation_two(ops, dt, L, N, H, dils):
    """As layers of 2 N sequences and half the steps, where their slices fit."""
    _against_levels(ops, dt, L, N, H, dils, 5)


@pytest.mark.parametrize("N,H,dils", [(17, 256, [1]), (40, 64, [1, 2]), (256, 256, [1, 2, 4, 8, 16, 32]), (90, 128, [4, 1, 2])])
def test_schedule_5_is_the_kernel_without_clusters(ops, monkeypatch, N, H, dils):
    """A refused launch is its error there, and not the generic kernel's result, so that the comparisons above are of this kernel."""
    from fractaltensor_b200._lib import FtbError
    D = len(dils)
    Wp = torch.zeros(D, 4 * H, 2 * H, dtype=torch.float16, device="cuda")
    x = torch.zeros(5, N, H, dtype=torch.float16, device="cuda")
    ops.lstm_dilated(x, Wp, dils, schedule=5)
    monkeypatch.setenv("FTB_REFUSE_COOPERATIVE", "1")
    with pytest.raises(FtbError) as e:
        ops.lstm_dilated(x, Wp, dils, schedule=5)
    assert e.value.code == 5
    ops.lstm_dilated(x, Wp, dils)  # the automatic choice falls back
    monkeypatch.undo()
    ops.check_status()


def test_schedule_5_where_it_does_not_apply(ops):
    """No layer of dilation 1: the generic persistent kernel, as for schedule 2."""
    _against_levels(ops, torch.float16, 9, 40, 128, [2, 3], 5)


def _against_levels(ops, dt, L, N, H, dils, schedule):
    D = len(dils)
    g = torch.Generator(device="cuda").manual_seed(N + L)
    u = lambda *s: ((torch.rand(*s, device="cuda", generator=g) * 2 - 1) / H ** 0.5).to(dt)
    Wp, b = ops.lstm_pack_weights(u(D, 4, H, H), u(D, 4, H, H), u(D, 4, H))
    x = torch.randn(L, N, H, device="cuda", generator=g).to(dt)
    ref, ref_c = ops.lstm_dilated(x, Wp, dils, b, schedule=1)
    for _ in range(3):
        h, c = ops.lstm_dilated(x, Wp, dils, b, schedule=schedule)
        ops.check_status()
        assert torch.equal(h, ref)
        for l, d in enumerate(dils):
            rows = min(d, L) * N
            cl, rl = c.view(D, -1, H)[l], ref_c.view(D, -1, H)[l]
            assert torch.equal(cl[:rows], rl[:rows])
