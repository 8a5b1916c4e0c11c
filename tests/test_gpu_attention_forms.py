"""Both forms of the attention kernel (CTAs of 256 query rows; of 128 rows whose slots take half of the keys each) on the
same calls: a rule on the number of query tiles chooses between them, so that calls small enough for a closed form would
else meet one of them only.  And chains of calls that feed one another: every form is launched as a dependent."""
import math

import pytest
import torch

from oracle import dense

pytestmark = pytest.mark.gpu
FORMS = [1, 2]


def attention(q, k, v, scale, form, causal=False, window=None, local=None, out=None):
    from fractaltensor_b200 import ops
    from fractaltensor_b200.ops import _dtype_code, _ptr, _stream, check, lib
    B, heads, S, d = q.shape
    out = torch.empty_like(q) if out is None else out
    left, right = local if local is not None else (window - 1 if window is not None else -1, 0)
    ws = ops.workspace(q.device)
    check(lib.ftb_flash_attn_form_fwd(_ptr(q), _ptr(k), _ptr(v), _ptr(out), B, heads, S, d, int(causal or local is not None),
                                      left, right, form, scale, _dtype_code(q), _ptr(ws), ws.numel(), _stream()),
          "ftb_flash_attn_form_fwd")
    return out


def _tolerance(dt):
    # P and the result are rounded to 16 bits (relative 2^-11 or 2^-8 each, averaged over the keys)
    return 1e-3 if dt == torch.float16 else 8e-3


def _close(out, ref, dt):
    out, ref = out.double().cpu(), ref.double()
    assert ((out - ref).norm() / ref.norm()).item() <= _tolerance(dt)
    assert (out - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("S,mask", [
    (256, {}), (512, {}), (1280, {}),
    (256, dict(causal=True)), (1024, dict(causal=True)), (1280, dict(causal=True)),
    # windows that begin at, before and behind the edge of a block and of 256 rows
    *[(1024, dict(causal=True, window=w)) for w in (1, 127, 128, 129, 255, 256, 257, 300, 1024, 5000)],
    *[(1280, dict(local=lr)) for lr in ((0, 0), (0, 127), (128, 128), (129, 1), (70, 300), (255, 256), (1000, 40), (3000, 3000))],
])
def test_both_forms_match_closed_form(dt, S, mask):
    from fractaltensor_b200 import ops
    q, k, v = dense.make_attention_inputs(1, 2, S, 128, S + len(mask), dtype=dt)
    sc = 1.0 / math.sqrt(128.0)
    ref = dense.attention_plain(q.double(), k.double(), v.double(), scale=sc, **mask)
    dev = [t.cuda() for t in (q, k, v)]
    outs = [attention(*dev, sc, form, **mask) for form in FORMS]
    ops.check_status()
    for out in outs:
        _close(out, ref, dt)
    assert torch.equal(attention(*dev, sc, 0, **mask), ops.flash_attention(*dev, scale=sc, **mask))


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("mask", [{}, dict(causal=True), dict(causal=True, window=400), dict(local=(300, 200))])
def test_maximum_that_moves_in_every_block(form, dt, mask):
    """Scores that rise by 11.5 powers of two a block: every block rescales the accumulator (2^8 is the threshold)."""
    from fractaltensor_b200 import ops
    S = 1024
    q, k, v = dense.make_attention_inputs(1, 1, S, 128, 3, dtype=dt)
    q, k = q * 0.125, k * 0.125
    q[..., 0], k[..., 0] = 1.0, torch.arange(S, dtype=torch.float32).to(dt) // 64 * 4
    out = attention(q.cuda(), k.cuda(), v.cuda(), 1.0, form, **mask)
    ops.check_status()
    _close(out, dense.attention_plain(q.double(), k.double(), v.double(), scale=1.0, **mask), dt)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("heads,S", [(3, 512), (40, 1024)])
def test_chain_of_dependent_calls(form, causal, heads, S):
    """Each call may be scheduled while the one before it drains and reads what that wrote: as queries, keys and values
    in turn, and into buffers that the call before still reads."""
    from fractaltensor_b200 import ops
    q, k, v = (t.cuda() for t in dense.make_attention_inputs(1, heads, S, 128, 4, dtype=torch.float16))
    call = lambda *a, **kw: attention(*a, 0.5, form, causal=causal, **kw)

    def chain(between):
        x = q
        for i in range(9):
            x = call(*((x, k, v), (q, x, v), (q, k, x))[i % 3])
            between()
        return x

    slow = chain(torch.cuda.synchronize)
    assert torch.isfinite(slow).all() and slow.abs().max().item() > 1e-3
    for _ in range(3):
        assert torch.equal(chain(lambda: None), slow)
    bufs = [v.clone(), torch.empty_like(v)]
    want = v
    for i in range(6):
        call(q, k, bufs[i & 1], out=bufs[(i + 1) & 1])
    for i in range(6):
        want = call(q, k, want)
        torch.cuda.synchronize()
    assert torch.equal(bufs[0], want)
    ops.check_status()


@pytest.mark.parametrize("form", FORMS)
def test_chain_in_a_cuda_graph(form):
    """The dependent launches become programmatic edges of the graph: a neighbour of another kernel at each end."""
    from fractaltensor_b200 import ops
    q, k, v = (t.cuda() for t in dense.make_attention_inputs(1, 16, 1024, 128, 5, dtype=torch.bfloat16))
    x, y, z = (torch.empty_like(q) for _ in range(3))

    def links():
        torch.mul(q, 0.5, out=x)
        attention(x, k, v, 0.5, form, causal=True, out=y)
        attention(q, y, v, 0.5, form, out=x)
        attention(q, k, x, 0.5, form, causal=True, out=y)
        torch.add(y, v, out=z)

    links()
    torch.cuda.synchronize()
    want = z.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        links()
    for _ in range(3):
        for t in (x, y, z):
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(z, want)
    ops.check_status()
