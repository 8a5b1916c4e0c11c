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
