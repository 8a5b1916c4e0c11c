"""Flash attention whose CTAs take 128 query rows and half of their key/value blocks a slot (csrc/flash_attn.cu,
kHalves): calls of few query tiles, against the closed form; walks of one block, of odd and of even numbers."""
import math

import pytest
import torch

from oracle import dense

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from fractaltensor_b200 import ops as _ops
    return _ops


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,heads,S,mask", [
    (1, 1, 256, {}),                                 # one block a slot
    (1, 2, 512, {}),
    (2, 3, 1280, {}),                                # ten blocks
    (1, 16, 2048, dict(causal=True)),                # walks of 1 to 16 blocks; the first leaves slot 1 empty
    (1, 2, 1024, dict(causal=True)),
    (1, 2, 1024, dict(causal=True, window=1)),       # one key a query
    (1, 2, 1536, dict(causal=True, window=200)),     # walks of two and three blocks, masked at both ends
    (1, 2, 1280, dict(local=(70, 300))),
    (1, 1, 768, dict(local=(0, 0))),
    (1, 3, 2048, dict(local=(1000, 40))),
    (1, 10, 4096, {}),                               # more CTAs than SMs
])
def test_matches_closed_form(ops, dt, B, heads, S, mask):
    q, k, v = (t.cuda() for t in dense.make_attention_inputs(B, heads, S, 128, S + heads, dtype=dt))
    sc = 1.0 / math.sqrt(128.0)
    out = ops.flash_attention(q, k, v, scale=sc, **mask)
    again = ops.flash_attention(q, k, v, scale=sc, **mask)
    ops.check_status()
    assert torch.equal(out, again)
    for b, h in {(0, 0), (B - 1, heads - 1)}:
        one = [t[b:b + 1, h:h + 1].cpu().double() for t in (q, k, v)]
        ref = dense.attention_plain(*one, scale=sc, **mask)
        got = out[b:b + 1, h:h + 1].double().cpu()
        # P and the result are rounded to 16 bits (relative 2^-11 or 2^-8 each, averaged over the keys)
        assert ((got - ref).norm() / ref.norm()).item() <= (1e-3 if dt == torch.float16 else 8e-3)
        assert (got - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())


def test_one_half_dominates(ops):
    """A key whose scores exceed all others by far, in either half: the other half's weight vanishes and nothing overflows."""
    for at in (100, 900):
        q, k, v = dense.make_attention_inputs(1, 2, 1024, 128, 5, dtype=torch.float16)
        k[:, :, at] *= 30
        out = ops.flash_attention(q.cuda(), k.cuda(), v.cuda(), scale=1.0)
        ops.check_status()
        ref = dense.attention_plain(q.double(), k.double(), v.double(), scale=1.0)
        assert (out.double().cpu() - ref).abs().max().item() <= 2e-2


def test_nan_stays_in_its_rows(ops):
    q, k, v = dense.make_attention_inputs(1, 2, 1024, 128, 6, dtype=torch.float16)
    q[0, 0, 300] = float("nan")
    v[0, 1, 900] = float("nan")
    bad = torch.isnan(ops.flash_attention(q.cuda(), k.cuda(), v.cuda(), scale=0.1, causal=True)).cpu()
    ops.check_status()
    rows = torch.zeros(1024, dtype=torch.bool)
    rows[300] = True
    assert bad[0, 0].any(-1).equal(rows)
    # (a masked key of a walked block has weight 0, and 0 times NaN is NaN, in both forms of the kernel)
    assert bad[0, 1, 900:].any(-1).all() and not bad[0, 1, :896].any()


def test_no_key_scores_above_minus_infinity_in_a_half(ops):
    """Keys of one half whose scores are all -inf count nothing beside the other half's."""
    q, k, v = dense.make_attention_inputs(1, 1, 512, 128, 7, dtype=torch.float16)
    q, k = q.abs(), k.clone()
    ref = dense.attention_plain(q.double(), k[:, :, :256].double(), v[:, :, :256].double(), scale=0.05)
    k[:, :, 256:] = float("-inf")
    out = ops.flash_attention(q.cuda(), k.cuda(), v.cuda(), scale=0.05)
    ops.check_status()
    assert (out.double().cpu() - ref).abs().max().item() <= 2e-2


@pytest.mark.parametrize("mask", [{}, dict(causal=True), dict(causal=True, window=300), dict(local=(200, 130))])
def test_scores_far_below_zero(ops, mask):
    """Finite scores of -2^106 and one key of -2^105 in bf16: the key whose score is the largest takes all the weight where
    a query sees it, elsewhere the visible keys share it.  (Powers of two: their product with the scale is exact.)"""
    S, top = 1024, 600
    v = dense.make_attention_inputs(1, 1, S, 128, 8, dtype=torch.bfloat16)[2]
    q, k = torch.zeros_like(v), torch.zeros_like(v)
    q[..., 0], k[..., 0], k[:, :, top, 0] = 2.0 ** 53, -2.0 ** 53, -2.0 ** 52
    out = ops.flash_attention(q.cuda(), k.cuda(), v.cuda(), scale=1.0, **mask).double().cpu()
    ops.check_status()
    ref = dense.attention_plain(q.double(), k.double(), v.double(), scale=1.0, **mask)
    # the result is rounded to 8 bits; P, a power of two or equal for all keys, is not in error
    assert (out - ref).abs().max().item() <= 2.0 ** -8 * ref.abs().max().item()
