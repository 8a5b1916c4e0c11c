"""Flash attention on pairs of CTAs (csrc/flash_pair.cu), named as form 3: masks and edges against the closed form, several
units of 256 rows a pair, references that move, what is not finite, and calls behind one another."""
import math

import pytest
import torch

from oracle import dense
from test_gpu_attention_forms import _close, attention

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("heads,S,mask", [
    (1, 256, {}), (2, 512, {}), (1, 1280, {}),
    (1, 256, dict(causal=True)), (2, 1024, dict(causal=True)), (1, 1280, dict(causal=True)),
    # windows in which a CTA of the pair begins a block late, ends a block early, or both
    *[(1, 1024, dict(causal=True, window=w)) for w in (1, 2, 127, 128, 129, 255, 256, 257, 300, 1024, 5000)],
    *[(1, 1280, dict(local=lr)) for lr in ((0, 0), (0, 127), (128, 128), (129, 1), (70, 300), (255, 256), (1000, 40), (3000, 3000))],
    # more units than pairs of SMs: two and three a pair, of different lengths, and (batch, head) entries in several groups
    (90, 256, {}), (200, 256, dict(causal=True)), (45, 1024, dict(causal=True)), (45, 1024, dict(causal=True, window=200)),
    (30, 1280, dict(local=(300, 200))),
])
def test_matches_closed_form(dt, heads, S, mask):
    from fractaltensor_b200 import ops
    q, k, v = dense.make_attention_inputs(1, heads, S, 128, S + len(mask), dtype=dt)
    sc = 1.0 / math.sqrt(128.0)
    dev = [t.cuda() for t in (q, k, v)]
    out = attention(*dev, sc, 3, **mask)
    again = attention(*dev, sc, 3, **mask)
    ops.check_status()
    assert torch.equal(out, again)
    for h in sorted({0, heads // 2, heads - 1}):
        one = [t[:, h:h + 1].double() for t in (q, k, v)]
        _close(out[:, h:h + 1], dense.attention_plain(*one, scale=sc, **mask), dt)


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("step", [4, -4])
@pytest.mark.parametrize("mask", [{}, dict(causal=True), dict(causal=True, window=400), dict(local=(300, 200))])
def test_maximum_that_moves_in_every_block(dt, step, mask):
    """Scores that rise (or fall) by 11.5 powers of two a block: every block moves the reference (2^8 is the threshold)."""
    from fractaltensor_b200 import ops
    S = 1024
    q, k, v = dense.make_attention_inputs(1, 1, S, 128, 3, dtype=dt)
    q, k = q * 0.125, k * 0.125
    q[..., 0], k[..., 0] = 1.0, torch.arange(S, dtype=torch.float32).to(dt) // 64 * step
    out = attention(q.cuda(), k.cuda(), v.cuda(), 1.0, 3, **mask)
    ops.check_status()
    _close(out, dense.attention_plain(q.double(), k.double(), v.double(), scale=1.0, **mask), dt)


def test_nan_stays_in_its_rows():
    """A NaN of V in the last block reaches none of the rows that do not walk it, though they share their MMAs with rows that do."""
    from fractaltensor_b200 import ops
    q, k, v = dense.make_attention_inputs(1, 2, 1024, 128, 6, dtype=torch.float16)
    q[0, 0, 300] = float("nan")
    v[0, 1, 900] = float("nan")
    for mask, first in (dict(causal=True), 896), (dict(local=(10, 0)), 896):
        bad = torch.isnan(attention(q.cuda(), k.cuda(), v.cuda(), 0.1, 3, **mask)).cpu()
        rows = torch.zeros(1024, dtype=torch.bool)
        rows[300] = True
        assert bad[0, 0].any(-1).equal(rows)
        assert bad[0, 1, 900].any() and not bad[0, 1, :first].any()
    # and at the other end: rows 128.. of the first pair do not walk block 0 with this window
    v[0, 1, 900] = 0.0
    v[0, 1, 5] = float("nan")
    bad = torch.isnan(attention(q.cuda(), k.cuda(), v.cuda(), 0.1, 3, local=(0, 100))).cpu()
    ops.check_status()
    assert bad[0, 1, 5].any() and not bad[0, 1, 128:].any()


def test_negative_scale_without_a_mask():
    """Taken as it was: the reference is then the smallest of a row's exponents, whose range the inputs keep small."""
    from fractaltensor_b200 import ops
    q, k, v = dense.make_attention_inputs(1, 2, 512, 128, 9, dtype=torch.float16)
    out = attention(q.cuda(), k.cuda(), v.cuda(), -0.05, 3)
    ops.check_status()
    _close(out, dense.attention_plain(q.double(), k.double(), v.double(), scale=-0.05), torch.float16)


@pytest.mark.parametrize("mask", [{}, dict(causal=True), dict(causal=True, window=300), dict(local=(200, 130))])
def test_scores_far_below_zero(mask):
    """As in the other forms: finite scores of -2^106 and one key of -2^105 in bf16."""
    from fractaltensor_b200 import ops
    S, top = 1024, 600
    v = dense.make_attention_inputs(1, 1, S, 128, 8, dtype=torch.bfloat16)[2]
    q, k = torch.zeros_like(v), torch.zeros_like(v)
    q[..., 0], k[..., 0], k[:, :, top, 0] = 2.0 ** 53, -2.0 ** 53, -2.0 ** 52
    out = attention(q.cuda(), k.cuda(), v.cuda(), 1.0, 3, **mask).double().cpu()
    ops.check_status()
    ref = dense.attention_plain(q.double(), k.double(), v.double(), scale=1.0, **mask)
    assert (out - ref).abs().max().item() <= 2.0 ** -8 * ref.abs().max().item()


def test_chain_of_dependent_calls_and_a_graph():
    """Calls of this form between calls of the others, each reading what the one before wrote, plainly and as a graph."""
    from fractaltensor_b200 import ops
    q, k, v = (t.cuda() for t in dense.make_attention_inputs(1, 40, 1024, 128, 4, dtype=torch.float16))
    x, y = torch.empty_like(q), torch.empty_like(q)

    def links(between=lambda: None):
        for form, args, out, causal in ((3, (q, k, v), x, False), (3, (q, x, v), y, True), (1, (q, k, y), x, True), (3, (x, k, v), y, False),
                                        (2, (q, y, v), x, True), (3, (q, k, x), y, True), (3, (y, k, v), x, True)):
            attention(*args, 0.5, form, causal=causal, out=out)
            between()

    links(torch.cuda.synchronize)
    want = x.clone()
    for _ in range(3):
        links()
        assert torch.equal(x, want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        links()
    for _ in range(2):
        x.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(x, want)
    ops.check_status()
