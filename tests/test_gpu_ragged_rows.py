"""Batch-major ragged batches of the stacked LSTM in one call (ops.lstm_stacked_ragged): the packed entry point on rows
sorted and put back by hand, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from fractaltensor_b200 import ops as _ops
    return _ops


@pytest.mark.parametrize("dt", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D,I,H,lens", [
    (1, 64, 64, [1]),
    (2, 128, 128, [5, 9, 1, 9, 5, 2, 9]),             # equal lengths keep their order
    (1, 192, 64, [3, 1, 4, 1, 5, 9, 2, 6]),           # rows in and out of different widths
    (3, 256, 256, [7] * 20),                          # nothing to sort
    (2, 64, 64, list(range(40, 0, -1)) + list(range(1, 30))),
])
def test_same_bits_as_packed(ops, dt, D, I, H, lens):
    g = torch.Generator(device="cuda").manual_seed(len(lens) + H)
    u = lambda *s: ((torch.rand(*s, device="cuda", generator=g) * 2 - 1) / H ** 0.5).to(dt)
    Wp, b = ops.lstm_pack_weights(u(D, 4, I, H), u(D, 4, H, H), u(D, 4, H))
    x = torch.randn(sum(lens), I, device="cuda", generator=g).to(dt)
    order = sorted(range(len(lens)), key=lambda n: -lens[n])
    start = [sum(lens[:n]) for n in range(len(lens))]
    active = [sum(n > t for n in lens) for t in range(max(lens))]
    src = torch.tensor([start[order[r]] + t for t in range(len(active)) for r in range(active[t])], device="cuda")
    hs, _ = ops.lstm_stacked_varlen(x[src].contiguous(), active, Wp, b)
    ref = torch.empty(sum(lens), H, dtype=dt, device="cuda")
    ref[src] = hs[D - 1]
    for _ in range(2):
        out = ops.lstm_stacked_ragged(x, lens, Wp, b)
        ops.check_status()
        assert torch.equal(out, ref)


def test_refused(ops):
    g = torch.Generator(device="cuda").manual_seed(1)
    u = lambda *s: torch.rand(*s, device="cuda", generator=g)
    Wp, b = ops.lstm_pack_weights(u(1, 4, 64, 64), u(1, 4, 64, 64), u(1, 4, 64))
    x = torch.zeros(6, 64, device="cuda")
    for lens in ([3, 0, 3], [3, 2], [7, -1]):
        with pytest.raises(ValueError):
            ops.lstm_stacked_ragged(x, lens, Wp, b)


def test_rows_that_begin_anywhere(ops):
    """embs.data may be a slice of a larger buffer, at any element."""
    from fractaltensor_b200 import frontend
    H, lens = 64, [4, 6, 2]
    g = torch.Generator(device="cuda").manual_seed(2)
    u = lambda *s: ((torch.rand(*s, device="cuda", generator=g) * 2 - 1) / 8).half()
    ft = lambda t: frontend.FractalTensor.from_dense(t, 2)
    params = [ft(u(2, 4, H, H)), ft(u(2, 4, H, H)), ft(u(2, 4, 1, H))]
    buf = torch.empty(sum(lens) * H + 8, device="cuda", dtype=torch.float16)
    nest = [list(range(n)) for n in lens]
    outs = []
    for at in (0, 1):
        rows = buf[at:at + sum(lens) * H]
        rows.copy_(torch.linspace(-1, 1, rows.numel(), device="cuda").half())
        outs.append(frontend.stacked_lstm(frontend.FractalTensor(rows, nest, (1, H)), *params))
        ops.check_status()
    assert outs[0].indices == nest and outs[0].element_shape == (1, H)
    assert torch.equal(outs[0].data, outs[1].data)


def test_capture_is_refused(ops):
    """A graph would keep the address of tables that end with the call.  (Nothing is replayed.)"""
    from fractaltensor_b200._lib import FtbError
    g = torch.Generator(device="cuda").manual_seed(3)
    u = lambda *s: (torch.rand(*s, device="cuda", generator=g) - 0.5).half()
    Wp, b = ops.lstm_pack_weights(u(1, 4, 64, 64), u(1, 4, 64, 64), u(1, 4, 64))
    x, lens = u(8, 64), [3, 5]
    want = ops.lstm_stacked_ragged(x, lens, Wp, b)
    torch.cuda.synchronize()
    graph, extra = torch.cuda.CUDAGraph(), torch.zeros(1, device="cuda")
    with torch.cuda.graph(graph):
        with pytest.raises(FtbError):
            ops.lstm_stacked_ragged(x, lens, Wp, b)
        extra.add_(1)  # the capture goes on
    del graph
    assert torch.equal(ops.lstm_stacked_ragged(x, lens, Wp, b), want)
    ops.check_status()


@pytest.mark.parametrize("dt", [torch.float32, torch.float16])
def test_row_tables_are_the_call_s_own(ops, dt):
    """Another host thread's call on the stream would put its tables where the stream's workspace has them: nothing of
    the rows is there.  The C entry without scratch, which has them there, gives the same bits."""
    from fractaltensor_b200.ops import _dtype_code, _ptr, _stream, check, ctypes, lib
    D, H, lens = 2, 64, [3, 9, 4, 9, 1]
    N, L, T = len(lens), max(lens), sum(lens)
    g = torch.Generator(device="cuda").manual_seed(4)
    u = lambda *s: (torch.rand(*s, device="cuda", generator=g) - 0.5).to(dt)
    Wp, b = ops.lstm_pack_weights(u(D, 4, H, H), u(D, 4, H, H), u(D, 4, H))
    x = u(T, H)
    packed = lib.ftb_lstm_stacked_varlen_workspace_bytes(D, L)
    room = lib.ftb_lstm_stacked_ragged_workspace_bytes(D, L, N)
    assert room >= packed + lib.ftb_lstm_stacked_ragged_scratch_bytes(L, N)
    ws = ops.workspace("cuda", room)
    rest = ws[packed:]
    rest.fill_(0xA5)
    got = ops.lstm_stacked_ragged(x, lens, Wp, b)
    ops.check_status()
    same = bool((rest == 0xA5).all())
    rest.zero_()
    assert same
    xt, out = torch.empty_like(x), torch.empty(T, H, dtype=dt, device="cuda")
    hs, c = torch.empty(D, T, H, dtype=dt, device="cuda"), torch.empty(D, N, H, device="cuda")
    args = (_ptr(x), _ptr(Wp), _ptr(b), (ctypes.c_int * N)(*lens), _ptr(xt), _ptr(hs), _ptr(c), _ptr(out), D, N, H, H,
            _dtype_code(x))
    check(lib.ftb_lstm_stacked_ragged_fwd(*args, _ptr(ws), room, _stream()), "ftb_lstm_stacked_ragged_fwd")
    ops.check_status()
    assert torch.equal(out, got)
    short = ctypes.c_size_t(lib.ftb_lstm_stacked_ragged_scratch_bytes(L, N) - 1)
    assert lib.ftb_lstm_stacked_ragged_fwd(*args, _ptr(ws), room - 1, _stream()) != 0
    assert lib.ftb_lstm_stacked_ragged_fwd_scratch(*args, _ptr(c), short, _ptr(ws), packed, _stream()) != 0
