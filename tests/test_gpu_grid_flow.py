"""Grid RNN with weights on chip and states that carry their own arrival (csrc/grid_flow.cu): bit for bit the result of one
launch per anti-diagonal, in every form and in the one that the automatic choice takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from fractaltensor_b200 import ops as _ops
    return _ops


def _inputs(ops, D, A, B, N, H, dt, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = lambda *s: ((torch.rand(*s, device="cuda", generator=g) * 2 - 1) / 8).to(dt)
    X, Y = (torch.randn(A, B, N, H, device="cuda", generator=g).to(dt) for _ in range(2))
    Wx, Wy = (ops.grid_pack_weights(u(D, 2 * H, H), u(D, H, H)) for _ in range(2))
    return X, Y, Wx, Wy, u(D, H).float(), u(D, H).float()


def _form(ops, args, nb, hx, hy):
    from fractaltensor_b200._lib import check, lib
    X, Wx = args[0], args[2]
    A, B, N, H = X.shape
    D = Wx.shape[0]
    ws = ops.workspace(X.device, lib.ftb_grid_rnn_workspace_bytes(D, A, B))
    check(lib.ftb_grid_flow_form_fwd(*(ops._ptr(t) for t in args), ops._ptr(hx), ops._ptr(hy), D, A, B, N, H, ops._dtype_code(X), nb,
                                     ops._ptr(ws), ws.numel(), ops._stream()), "ftb_grid_flow_form_fwd")
    ops.check_status()


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D,A,B,N,H", [
    (1, 1, 1, 1, 64),      # one cell: nobody waits for anything
    (1, 1, 20, 5, 256),    # one row: h_y alone
    (1, 20, 1, 5, 256),    # one column: h_x alone
    (2, 3, 8, 16, 128),    # whole slices; the fill's count ends with the columns
    (1, 4, 17, 33, 192),   # a half tile of units in the second CTA of a pair; a slice of one sequence; past the fill's lead
    (3, 5, 9, 64, 64),     # a tile of 64 units
    (2, 40, 24, 20, 256),  # more chains than groups: weights change from chain to chain
    (1, 90, 3, 70, 128),   # chains shorter than the fill's lead, several of them ahead
])
def test_same_bits_as_levels(ops, dt, D, A, B, N, H):
    args = _inputs(ops, D, A, B, N, H, dt, D * 100 + N)
    rx, ry = ops.grid_rnn(*args, schedule=1)
    hx, hy = ops.grid_rnn(*args)
    ops.check_status()
    assert torch.equal(hx, rx) and torch.equal(hy, ry)
    for nb in (16, 32, 64):
        # what the buffers held before (states of another call, all of them valid) must not be taken for an arrival
        hx, hy = torch.randn_like(rx), torch.randn_like(ry)
        for _ in range(2):
            _form(ops, args, nb, hx, hy)
            assert torch.equal(hx, rx) and torch.equal(hy, ry)


@pytest.mark.parametrize("D,A,B,N,H", [(1, 6, 9, 40, 256), (3, 7, 20, 70, 128), (2, 5, 8, 33, 192)])
def test_workspaces_of_every_size(ops, D, A, B, N, H):
    """What a call asks for, room for the counters of wider slices alone, for the tables alone, and for neither."""
    from fractaltensor_b200._lib import check, lib
    args = _inputs(ops, D, A, B, N, H, torch.float16, N)
    rx, ry = ops.grid_rnn(*args, schedule=1)
    tables, full = lib.ftb_grid_rnn_tables_bytes(D, A, B), lib.ftb_grid_rnn_call_workspace_bytes(D, A, B, N, H, 1)
    for size in (full, tables + (full - tables) // 2, tables + 4, tables, lib.ftb_workspace_bytes()):
        hx, hy = torch.randn_like(rx), torch.randn_like(ry)
        room = torch.zeros(size + 256, dtype=torch.uint8, device="cuda")
        room[size:] = 77  # behind the workspace: not the call's
        check(lib.ftb_grid_rnn_fwd(*(ops._ptr(t) for t in args), ops._ptr(hx), ops._ptr(hy), D, A, B, N, H, 1, ops._ptr(room), size,
                                   ops._stream()), "ftb_grid_rnn_fwd")
        torch.cuda.synchronize()
        assert int(room[:4].view(torch.int32)) == 0 and bool((room[size:] == 77).all())
        assert torch.equal(hx, rx) and torch.equal(hy, ry), size


def test_nan_states_are_states(ops):
    """A NaN state (0x7FFF) is a value like any other, also where an input has the fill pattern's bits."""
    X, Y, Wx, Wy, bx, by = _inputs(ops, 1, 5, 6, 20, 128, torch.float16)
    X[1, 2, 3] = float("nan")
    X.view(torch.int16)[1, 2, 4] = -1
    rx, ry = ops.grid_rnn(X, Y, Wx, Wy, bx, by, schedule=1)
    for nb in (16, 32, 64):
        hx, hy = torch.empty_like(rx), torch.empty_like(ry)
        _form(ops, (X, Y, Wx, Wy, bx, by), nb, hx, hy)
        for a, b in ((hx, rx), (hy, ry)):
            assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.nan_to_num(a), torch.nan_to_num(b))
    assert torch.isnan(rx[0, 2:, 2:, 3:5]).all() and not torch.isnan(rx[0, 0]).any() and not torch.isnan(rx[:, :, :, 5:]).any()


def test_forms_that_do_not_exist(ops):
    args = _inputs(ops, 1, 2, 2, 600, 64, torch.float16)
    hx = torch.empty(1, 2, 2, 600, 64, dtype=torch.float16, device="cuda")
    for nb in (8, 48, 128, 16):  # 16: more slices than there are counters for
        with pytest.raises(RuntimeError):
            _form(ops, args, nb, hx, torch.empty_like(hx))


@pytest.mark.parametrize("D,A,B,N,H", [
    (1, 2, 3, 2049, 64), (2, 2, 2, 2300, 256),     # more than 32 slices of 64
    (1, 2, 5, 4096, 64), (1, 2, 5, 4097, 64),      # the last batch that has counters, the first that has none
    (2, 30, 1, 1100, 256), (3, 12, 2, 1200, 192),  # a few columns, many chains: the generic wavefront by the rule
    (2, 30, 5, 300, 256),                          # one column more
])
def test_large_batches(ops, D, A, B, N, H):
    args = _inputs(ops, D, A, B, N, H, torch.bfloat16, N)
    rx, ry = ops.grid_rnn(*args, schedule=1)
    hx, hy = ops.grid_rnn(*args)
    ops.check_status()
    assert torch.equal(hx, rx) and torch.equal(hy, ry)


def test_many_short_chains_do_not_take_long(ops):
    """Rows of one column and a large batch: the generic wavefront's 0.13 ms, not the 0.27 of one chain behind another."""
    args = _inputs(ops, 3, 14, 1, 1715, 192, torch.float16)
    took = {0: [], 2: []}
    for _ in range(8):  # in turn, so that both meet the same clocks
        for schedule in (0, 2):
            ops.grid_rnn(*args, schedule=schedule)
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            for _ in range(4):
                ops.grid_rnn(*args, schedule=schedule)
            end.record()
            end.synchronize()
            took[schedule].append(start.elapsed_time(end))
    assert min(took[0]) < 1.2 * min(took[2]), took
