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


def test_a_full_launch_queue_does_not_stop_other_threads():
    """More calls than a stream's queue holds, behind 0.6 s of waiting: the thread that makes them stands still
    until the queue moves, the other threads of the program do not."""
    import threading
    import time
    from fractaltensor_b200 import ops
    A, B, C = _b2b()
    out = ops.b2b_gemm(A, B, C)
    torch.cuda.synchronize()
    took = []

    def many_calls():
        torch.cuda._sleep(int(0.6 * 1.9e9))
        t0 = time.perf_counter()
        for _ in range(4000):
            ops.b2b_gemm(A, B, C, out)
        took.append(time.perf_counter() - t0)

    caller = threading.Thread(target=many_calls)
    gap, last = 0.0, time.perf_counter()
    caller.start()
    while caller.is_alive():
        time.sleep(0.002)
        now = time.perf_counter()
        gap, last = max(gap, now - last), now
    torch.cuda.synchronize()
    assert took[0] > 0.4  # the queue was full
    assert gap < 0.25


def test_an_error_of_the_library_is_raised_without_a_second_call(monkeypatch):
    from fractaltensor_b200 import ops
    from fractaltensor_b200._lib import FtbError
    ops.b2b_gemm(*_b2b())
    again = []
    for name in ("ftb_b2b_gemm", "ftb_flash_attn_fwd", "ftb_flash_attn_window_fwd", "ftb_sparse_attn_fwd"):
        monkeypatch.setattr(ops.lib, name, lambda *a, name=name: again.append(name) or 0)
    z = lambda *s: torch.zeros(*s, device="cuda", dtype=torch.half)
    for where, call in (("ftb_b2b_gemm", lambda: ops.b2b_gemm(z(1, 100, 64), z(1, 128, 64), z(1, 64, 128))),
                        ("ftb_flash_attn_fwd", lambda: ops.flash_attention(z(1, 1, 100, 128), *[z(1, 1, 100, 128)] * 2)),
                        ("ftb_flash_attn_window_fwd", lambda: ops.flash_attention(*[z(1, 1, 256, 128)] * 3, causal=True, window=0)),
                        ("ftb_sparse_attn_fwd", lambda: ops.sparse_attention(*[z(1, 1, 64, 48)] * 3, None))):
        with pytest.raises(FtbError, match=where) as e:
            call()
        assert e.value.code == 1
    assert again == []


@pytest.mark.parametrize("dt", [torch.float16, torch.float32])
def test_calls_of_the_word_program_through_python_and_native(monkeypatch, dt):
    """The same results through the native front and through the Python checks, and the same errors."""
    from fractaltensor_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(5)
    r = lambda *s: (torch.randn(*s, device="cuda", generator=g) * 0.1).to(dt)
    D, H, V, lens = 2, 64, 2008, [3, 7, 1, 7]
    T = sum(lens)
    table, ids = r(50, H), torch.randint(0, 50, (T,), device="cuda", generator=g)
    W, U, b, P = r(D, 4, H, H), r(D, 4, H, H), r(D, 4, 1, H), r(H, V)

    def program():
        x = ops.embedding_gather(table, ids)
        Wp, bias = ops.lstm_pack_weights(W, U, b)
        Wp0, none = ops.lstm_pack_weights(W, U)
        h = ops.lstm_stacked_ragged(x, lens, Wp, bias)
        return [x, Wp, bias, Wp0, h, ops.lstm_stacked_ragged(x, lens, Wp)] + ([ops.project_softmax_rows(h, P)] if dt != torch.float32 else []), none

    def errors():
        x, (Wp, bias) = ops.embedding_gather(table, ids), ops.lstm_pack_weights(W, U, b)
        out = []
        for call in (lambda: ops.embedding_gather(table, ids.int()), lambda: ops.embedding_gather(table, ids, x[1:]),
                     lambda: ops.lstm_pack_weights(W, U[:1], b), lambda: ops.lstm_pack_weights(W, U, b[:1]),
                     lambda: ops.lstm_stacked_ragged(x, [3, 7, 1], Wp, bias), lambda: ops.lstm_stacked_ragged(x, [3, 8, 0, 7], Wp, bias),
                     lambda: ops.lstm_stacked_ragged(x, lens, Wp, bias[:, 1:]), lambda: ops.lstm_stacked_ragged(x[:, ::2], lens, Wp, bias),
                     lambda: ops.project_softmax_rows(x, P[:32])):
            with pytest.raises(Exception) as e:
                call()
            out.append(type(e.value))
        return out

    ops.embedding_gather(table, ids)  # (that call and the projection leave it to the Python checks to make a stream's first workspace)
    taken = {}

    def recorded(name):
        native_call = getattr(_lib.host, name)

        def call(*args):
            done = native_call(*args)
            taken.setdefault(name, []).append(done is not None and type(done) is not int)
            return done
        return call

    names = ["embedding_gather", "lstm_pack_weights", "lstm_stacked_ragged"] + (["project_softmax"] if dt != torch.float32 else [])
    front = {name: staticmethod(recorded(name)) for name in names}
    monkeypatch.setattr(ops, "host", type("Host", (_lib._NoHost,), {"current_stream": staticmethod(_lib.host.current_stream), **front}))
    native, none = program()
    assert none is None
    # every one of them by the native front, not by the Python checks behind it
    assert taken == {"embedding_gather": [True], "lstm_pack_weights": [True, True], "lstm_stacked_ragged": [True, True],
                     **({"project_softmax": [True]} if dt != torch.float32 else {})}
    wrong = errors()
    ops.check_status()
    monkeypatch.setattr(ops, "host", type("Host", (_lib._NoHost,), {"current_stream": staticmethod(_lib.host.current_stream)}))
    plain, _ = program()
    assert all(torch.equal(a, b) for a, b in zip(native, plain)) and wrong == errors()
    ops.check_status()


def test_lengths_that_are_not_the_rows_cost_no_workspace():
    """Refused as they were by the Python checks, before the tables of the longest are made."""
    from fractaltensor_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(5)
    r = lambda *s: (torch.randn(*s, device="cuda", generator=g) * 0.1).half()
    x, (Wp, b) = r(18, 64), ops.lstm_pack_weights(r(3, 4, 64, 64), r(3, 4, 64, 64), r(3, 4, 64))
    ops.lstm_stacked_ragged(x, [3, 7, 1, 7], Wp, b)
    torch.cuda.synchronize()
    room, held = [w.numel() for w in ops._workspaces.values()], torch.cuda.memory_allocated()
    for lens in ([1000000], [17, 200000], [3, 7, 1], [2 ** 40], [18 + 2 ** 33, -2 ** 33], [-2, 20], [18, 0], [10 ** 9, 10 ** 9]):
        with pytest.raises(ValueError):
            ops.lstm_stacked_ragged(x, lens, Wp, b)
    with pytest.raises(ValueError):
        ops.lstm_stacked_ragged(x.reshape(2, 9, 64), [18], Wp, b)
    assert [w.numel() for w in ops._workspaces.values()] == room and torch.cuda.memory_allocated() <= held
