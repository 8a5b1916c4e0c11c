"""Calls on several streams of one device at a time: what a call keeps for itself while it runs must be
its own."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rnn_attention_inputs(seed, dt, Ls=24, Lt=9, N=33, H=256):
    from fractaltensor_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = lambda *s: ((torch.rand(*s, device="cuda", generator=g) * 2 - 1) / H ** 0.5).to(dt)
    src, trg = (torch.randn(n, N, H, device="cuda", generator=g).to(dt) for n in (Ls, Lt))
    return (src, trg, ops.rnn_pack_weights(u(H, H), u(H, H)), ops.rnn_pack_weights(u(H, H), u(H, H)), u(H).float(),
            u(H).float(), u(H), u(H))


def _together(calls, rounds=12):
    """Each of `calls` on a stream of its own, `rounds` times, started in turn -> the last results."""
    streams = [torch.cuda.Stream() for _ in calls]
    for s in streams:
        s.wait_stream(torch.cuda.current_stream())
    out = [None] * len(calls)
    for _ in range(rounds):
        for i, (s, call) in enumerate(zip(streams, calls)):
            with torch.cuda.stream(s):
                out[i] = call()
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_rnn_attention_leaves_the_shared_workspace_alone(dt):
    """The fp32 input halves of the encoder are the call's own: nothing behind the status word changes."""
    from fractaltensor_b200 import ops
    from fractaltensor_b200._lib import lib
    args = _rnn_attention_inputs(1, dt)
    ws = ops.workspace("cuda", 1 << 22)
    rest = ws[lib.ftb_workspace_bytes():]
    rest.fill_(0xA5)
    ops.rnn_attention(*args)
    ops.check_status()
    same = bool((rest == 0xA5).all())
    rest.zero_()
    assert same


def test_rnn_attention_on_two_streams():
    from fractaltensor_b200 import ops
    args = [_rnn_attention_inputs(s, torch.bfloat16) for s in (1, 2)]
    alone = [ops.rnn_attention(*a) for a in args]
    both = _together([lambda a=a: ops.rnn_attention(*a) for a in args])
    for one, other in zip(alone, both):
        assert all(torch.equal(a, b) for a, b in zip(one, other))
    ops.check_status()


@pytest.mark.parametrize("program", ["stacked", "fp32", "ragged", "dilated", "grid"])
def test_recurrent_programs_on_two_streams(program):
    """Tables and counters of a call are in the workspace of its stream."""
    from fractaltensor_b200 import ops

    def call(seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        dt = torch.float32 if program == "fp32" else torch.float16
        H, D, L, N = 128, 2, 24, 20
        u = lambda *s: ((torch.rand(*s, device="cuda", generator=g) * 2 - 1) / H ** 0.5).to(dt)
        r = lambda *s: torch.randn(*s, device="cuda", generator=g).to(dt)
        if program == "grid":
            X, Y = r(5, 6, N, H), r(5, 6, N, H)
            Wx, Wy = (ops.grid_pack_weights(u(1, 2 * H, H), u(1, H, H)) for _ in range(2))
            return lambda: ops.grid_rnn(X, Y, Wx, Wy)
        Wp, b = ops.lstm_pack_weights(u(D, 4, H, H), u(D, 4, H, H), u(D, 4, H))
        if program == "ragged":
            active = [N] * 5 + [9] * 6 + [2] * 3
            x = r(sum(active), H)
            return lambda: ops.lstm_stacked_varlen(x, active, Wp, b)
        x = r(L, N, H)
        if program == "dilated":
            return lambda: ops.lstm_dilated(x, Wp, [1, 2], b)[:1]
        return lambda: ops.lstm_stacked(x, Wp, b)

    calls = [call(s) for s in (1, 2)]
    alone = [c() for c in calls]
    both = _together(calls)
    ops.check_status()
    for one, other in zip(alone, both):
        assert all(torch.equal(a, b) for a, b in zip(one, other))


def test_workspaces_are_bounded_and_their_status_is_found(monkeypatch):
    from fractaltensor_b200 import ops
    from fractaltensor_b200._lib import FtbError
    monkeypatch.setattr(ops, "_workspaces", {})
    monkeypatch.setattr(ops, "_MAX_WORKSPACES", 3)
    seen = []
    for _ in range(5):
        with torch.cuda.stream(torch.cuda.Stream()):
            seen.append(ops.workspace("cuda"))
            assert ops.workspace("cuda") is seen[-1] and len(ops._workspaces) <= 3
    assert len({w.data_ptr() for w in seen[-3:]}) == 3
    torch.cuda.synchronize()
    seen[-1][:4].view(torch.int32).fill_(22)  # as a call on that stream would leave it
    torch.cuda.synchronize()
    with pytest.raises(FtbError):
        ops.check_status()
    ops.check_status()  # cleared


def test_the_handle_of_the_current_stream():
    from fractaltensor_b200._lib import _NoHost, host
    side = torch.cuda.Stream()
    for stream in (torch.cuda.current_stream(), side):
        with torch.cuda.stream(stream):
            for h in (host, _NoHost):
                assert h.current_stream(-1) == h.current_stream(0) == stream.cuda_stream


def test_a_capture_takes_a_workspace_that_is_there():
    from fractaltensor_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(1)
    A, B, C = (torch.randn(s, device="cuda", generator=g).half() * 0.1 for s in ((1, 128, 64), (1, 128, 64), (1, 64, 128)))
    ref = ops.b2b_gemm(A, B, C)
    before = dict(ops._workspaces)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        out = ops.b2b_gemm(A, B, C)
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, ref) and ops._workspaces == before


@pytest.mark.parametrize("program", ["varlen", "ragged", "stacked"])
def test_host_threads_on_one_stream(program):
    """Host threads share the default stream and so its workspace: the tables of one thread's call are not those of
    another's kernels."""
    import threading

    from fractaltensor_b200 import ops

    def call(seed, N):
        g = torch.Generator(device="cuda").manual_seed(seed)
        H, D, L = 64, 2, 20
        u = lambda *s: ((torch.rand(*s, device="cuda", generator=g) * 2 - 1) / H ** 0.5).half()
        Wp, b = ops.lstm_pack_weights(u(D, 4, H, H), u(D, 4, H, H), u(D, 4, H))
        if program == "stacked":
            x = u(L, N, H)
            return lambda: ops.lstm_stacked(x, Wp, b, schedule=2)[0]
        lens = [1 + (7 * n + seed) % L for n in range(N)]
        x = u(sum(lens), H)
        if program == "ragged":
            return lambda: ops.lstm_stacked_ragged(x, lens, Wp, b)
        active = [sum(n > t for n in lens) for t in range(max(lens))]
        return lambda: ops.lstm_stacked_varlen(x, active, Wp, b)[0]

    calls = [call(s, 5 + 9 * s) for s in range(4)]
    alone = [c() for c in calls]
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        for _ in range(40):
            if not torch.equal(calls[i](), alone[i]):
                wrong.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    ops.check_status()
    assert not wrong
