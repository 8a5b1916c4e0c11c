"""GPU parity of the token-level sparse attention (dilated window + random + global keys) with the
oracle and with the fixture the reference's frontend produced
(examples/sparse_attention/sparse_attention.py:24-76)."""
import os

import numpy as np
import pytest
import torch

from oracle import dense

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from fractaltensor_b200 import ops as _ops
    return _ops


def _load(golden_dir, name):
    z = np.load(os.path.join(golden_dir, name))
    return {k: (torch.from_numpy(z[k]) if z[k].ndim > 0 else z[k].item()) for k in z.files}


def _inputs(B, heads, S, d, ng, R, seed, dt):
    g = torch.Generator().manual_seed(seed)
    q, k, v = (torch.rand(B, heads, S, d, generator=g).to(dt) for _ in range(3))
    pos = torch.randint(0, S, (B, heads, S - 2 * ng, max(R, 1)), generator=g, dtype=torch.int32)[..., :R].contiguous()
    return q, k, v, pos


def test_sparse_attention_golden(ops, golden_dir):
    """What the reference's frontend returns for per_head_attn (softmax over dimension 0, as shipped)."""
    g = _load(golden_dir, "sparse_attention_small.npz")
    ws, dil = int(g["window_size"]), int(g["dilation"])
    q, k, v = (g[n][None, None].contiguous().cuda() for n in ("q", "k", "v"))
    pos = g["rand_pos"].to(torch.int32)[None, None].contiguous().cuda()
    out = ops.sparse_attention(q, k, v, pos, ws, dil, as_shipped=True)
    ops.check_status()
    assert (out[0, 0].cpu() - g["out"]).abs().max().item() <= 1e-5
    # the attention the example describes, against the oracle
    att = ops.sparse_attention(q, k, v, pos, ws, dil)
    ref = dense.sparse_attention_dense(g["q"].double(), g["k"].double(), g["v"].double(), g["rand_pos"], ws, dil)
    assert (att[0, 0].cpu().double() - ref).abs().max().item() <= 1e-5


def test_sparse_attention_frontend_nestings(ops, golden_dir):
    """The model-level signature: FractalTensors of [1, d] tokens, one head or [B][heads][S]."""
    from fractaltensor_b200 import frontend
    g = _load(golden_dir, "sparse_attention_small.npz")
    ws, dil = int(g["window_size"]), int(g["dilation"])
    S, d = g["q"].shape
    ft = lambda t, depth: frontend.FractalTensor.from_dense(t.cuda(), depth)
    one = frontend.sparse_attention(ft(g["q"][:, None], 1), ft(g["k"][:, None], 1), ft(g["v"][:, None], 1),
                                    ft(g["rand_pos"][:, None], 1), ws, dil, as_shipped=True)
    assert len(one) == S and one.element_shape == (1, d)
    assert (one.to_dense()[:, 0].cpu() - g["out"]).abs().max().item() <= 1e-5
    B, heads = 2, 3
    q, k, v, pos = _inputs(B, heads, S, d, 3, 3, 5, torch.float32)
    many = frontend.sparse_attention(ft(q[:, :, :, None], 3), ft(k[:, :, :, None], 3), ft(v[:, :, :, None], 3),
                                     ft(pos[:, :, :, None], 3), ws, dil)
    ops.check_status()
    assert many.depth == 3 and many.element_shape == (1, d)
    ref = dense.sparse_attention_dense(q.double(), k.double(), v.double(), pos, ws, dil)
    assert (many.to_dense()[:, :, :, 0].cpu().double() - ref).abs().max().item() <= 1e-5


CASES = [
    # B, heads, S, d, window, dilation, n_global, R
    (1, 1, 16, 64, 5, 2, 3, 3),      # the example's own sizes
    (2, 4, 64, 64, 5, 2, 3, 3),
    (1, 2, 33, 32, 1, 1, 0, 0),      # a window of the token itself, nothing else
    (1, 2, 40, 128, 7, 3, 1, 5),
    (2, 1, 50, 256, 3, 1, 4, 0),     # no random keys
    (1, 3, 128, 64, 31, 2, 16, 33),  # 64 keys per windowed token, 32 global keys
    (1, 1, 12, 64, 5, 2, 6, 2),      # every token is global
    (1, 2, 70, 64, 9, 4, 32, 1),     # 64 global keys: two per lane
    (2, 3, 300, 64, 5, 2, 3, 3),     # the example's key counts: interior tiles by the kernel built for them
    (1, 2, 300, 128, 5, 3, 2, 3),    # the same with dilation 3 and 128 elements per head
    (1, 2, 1000, 32, 5, 1, 0, 3),    # no global tokens, dilation 1
    (1, 1, 200, 256, 5, 2, 30, 3),   # 60 global keys, 256 elements per head
]


@pytest.mark.parametrize("dt", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shipped", [False, True])
@pytest.mark.parametrize("case", CASES)
def test_sparse_attention_matches_oracle(ops, dt, shipped, case):
    B, heads, S, d, ws, dil, ng, R = case
    q, k, v, pos = _inputs(B, heads, S, d, ng, R, S * 7 + d + R, dt)
    scale = 1.0 if shipped else 0.25
    out = ops.sparse_attention(q.cuda(), k.cuda(), v.cuda(), pos.cuda() if R else None, ws, dil, ng, scale=scale,
                               as_shipped=shipped)
    ops.check_status()
    ref = dense.sparse_attention_dense(q.double() * scale, k.double(), v.double(),
                                       pos if R else torch.zeros(B, heads, S - 2 * ng, 0, dtype=torch.int32), ws, dil,
                                       ng, as_shipped=shipped)
    # fp32 arithmetic everywhere; 16-bit types round the stored output once (2^-11 / 2^-8 relative)
    rel = {torch.float32: 2e-6, torch.float16: 6e-4, torch.bfloat16: 5e-3}[dt]
    err = (out.cpu().double() - ref).abs().max().item()
    assert err <= rel * max(1.0, ref.abs().max().item()), err


def test_sparse_attention_full_size(ops):
    """The sizes the example names for real use (sequence 4096, 16 heads of 64, batch 2), fp32, every
    token compared with the oracle; and the shipped form against a plain gather-and-sum."""
    B, heads, S, d, ws, dil, ng, R = 2, 16, 4096, 64, 5, 2, 3, 3
    q, k, v, pos = _inputs(B, heads, S, d, ng, R, 77, torch.float32)
    out = ops.sparse_attention(q.cuda(), k.cuda(), v.cuda(), pos.cuda(), ws, dil, ng, scale=0.125)
    ops.check_status()
    ref = dense.sparse_attention_dense(q * 0.125, k, v, pos, ws, dil, ng)
    assert (out.cpu() - ref).abs().max().item() <= 2e-5
    shipped = ops.sparse_attention(q.cuda(), k.cuda(), v.cuda(), pos.cuda(), ws, dil, ng, as_shipped=True)
    half = (ws - 1) * dil // 2
    i = torch.arange(ng, S - ng)
    win = i[:, None] - half + torch.arange(ws)[None, :] * dil
    win = torch.where(win < 0, win + S - 1, torch.where(win >= S, win - S, win))
    idx = torch.cat([win.expand(B, heads, -1, -1), pos.long()], dim=-1)            # [B, heads, S - 6, ws + R]
    total = torch.zeros(B, heads, S - 2 * ng, d)
    for j in range(ws + R):
        total += torch.gather(v, 2, idx[..., j, None].expand(-1, -1, -1, d))
    assert (shipped[:, :, ng:S - ng].cpu() - total).abs().max().item() <= 1e-5


def test_sparse_attention_bad_position_sets_status(ops):
    q, k, v, pos = _inputs(1, 1, 16, 64, 3, 3, 3, torch.float32)
    pos[0, 0, 4, 1] = 16
    out = ops.sparse_attention(q.cuda(), k.cuda(), v.cuda(), pos.cuda())
    torch.cuda.synchronize()
    assert torch.isfinite(out).all()
    from fractaltensor_b200._lib import FtbError
    with pytest.raises(FtbError) as e:
        ops.check_status()
    assert e.value.code == 22
    ops.check_status()  # the word was cleared by the failed check


def test_sparse_attention_rejects_host_tensors(ops):
    q, k, v, pos = _inputs(1, 1, 16, 64, 3, 3, 3, torch.float32)
    with pytest.raises(RuntimeError):
        ops.sparse_attention(q, k, v, pos)
    with pytest.raises(ValueError):
        ops.sparse_attention(q.cuda(), k.cuda(), v.cuda(), pos.cuda().long())


def test_sparse_attention_empty_batch_and_single_tile_edges(ops):
    """No heads at all is a no-op; a sequence of exactly one tile with every kind of token in it."""
    q = torch.empty(0, 4, 64, 64, device="cuda")
    pos = torch.empty(0, 4, 58, 3, dtype=torch.int32, device="cuda")
    out = ops.sparse_attention(q, q.clone(), q.clone(), pos)
    ops.check_status()
    assert out.shape == q.shape
    q, k, v, pos = _inputs(3, 2, 64, 64, 3, 3, 9, torch.float32)
    out = ops.sparse_attention(q.cuda(), k.cuda(), v.cuda(), pos.cuda())
    ops.check_status()
    ref = dense.sparse_attention_dense(q.double(), k.double(), v.double(), pos)
    assert (out.cpu().double() - ref).abs().max().item() <= 2e-6 * max(1.0, ref.abs().max().item())


@pytest.mark.parametrize("dt", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("case", [
    # interior tiles by the routine that is told the window: 1 to 4 random keys, windows 1 to 7
    (1, 2, 300, 64, 1, 1, 0, 1),
    (2, 1, 257, 128, 3, 3, 2, 2),
    (1, 2, 300, 32, 7, 2, 4, 3),
    (1, 1, 333, 256, 5, 1, 1, 4),
    (1, 2, 300, 64, 7, 3, 3, 5),     # one random key more: the general routine
    (1, 1, 300, 64, 9, 1, 3, 4),     # a wider window: the general routine
])
def test_sparse_attention_key_counts(ops, dt, case):
    test_sparse_attention_matches_oracle(ops, dt, False, case)


@pytest.mark.parametrize("dt", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,heads,S,d,window,dilation,ng,R", [
    (1, 1, 200, 32, 5, 2, 3, 3),       # one interior tile and a last one that is not full
    (2, 5, 333, 64, 7, 3, 1, 4),       # the most keys of the routine
    (1, 3, 1000, 128, 3, 1, 4, 1),
    (1, 40, 1500, 64, 5, 2, 3, 3),     # more tiles than CTAs: stages filled behind the last warp that has read them
    (1, 70, 700, 128, 5, 1, 2, 2),
    (1, 2, 130, 256, 1, 1, 0, 2),      # no global token, no window beyond the token itself
])
def test_interior_walk_matches_oracle(ops, dt, B, heads, S, d, window, dilation, ng, R):
    """Tiles of 1 to 4 random keys and windows up to 7 (positions and random rows requested a pass ahead) against the
    oracle, random positions at both ends of the sequence among them."""
    q, k, v, pos = _inputs(B, heads, S, d, ng, R, S + d, dt)
    pos[..., 0].view(-1)[::7] = 0
    pos[..., -1].view(-1)[::5] = S - 1
    sc = 1.0 / d ** 0.5
    out = ops.sparse_attention(q.cuda(), k.cuda(), v.cuda(), pos.cuda(), window, dilation, ng, sc)
    ops.check_status()
    for b, h in {(0, 0), (B - 1, heads - 1)}:
        ref = dense.sparse_attention_dense(q[b, h].double() * sc, k[b, h].double(), v[b, h].double(), pos[b, h], window, dilation, ng)
        assert (out[b, h].cpu().double() - ref).abs().max().item() <= (1e-5 if dt == torch.float32 else 1e-2)
    # every head is the program of that head alone
    one = ops.sparse_attention(q[-1:, -1:].cuda(), k[-1:, -1:].cuda(), v[-1:, -1:].cuda(), pos[-1:, -1:].cuda(), window,
                               dilation, ng, sc)
    assert torch.equal(one[0, 0], out[-1, -1])


def test_interior_walk_reports_positions_outside(ops):
    from fractaltensor_b200._lib import FtbError
    q, k, v, pos = _inputs(1, 2, 512, 64, 3, 3, 4, torch.float32)
    good = ops.sparse_attention(q.cuda(), k.cuda(), v.cuda(), pos.cuda(), 5, 2, 3, 1.0)
    ops.check_status()
    bad = pos.clone()
    bad[0, 1, 250, 1] = 512
    out = ops.sparse_attention(q.cuda(), k.cuda(), v.cuda(), bad.cuda(), 5, 2, 3, 1.0)
    with pytest.raises(FtbError):
        ops.check_status()
    same = torch.ones(512, dtype=torch.bool)
    same[253] = False
    assert torch.equal(out[0, 0], good[0, 0]) and torch.equal(out[0, 1][same.cuda()], good[0, 1][same.cuda()])


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("R", [1, 2, 3, 4])
@pytest.mark.parametrize("window", [1, 3, 5, 7])
def test_every_pair_of_key_counts(ops, dt, window, R):
    """Each pair of window and random keys that has a routine of its own, with interior and edge tiles."""
    test_interior_walk_matches_oracle(ops, dt, 1, 3, 261, 64, window, 2, 2, R)


@pytest.mark.parametrize("dt,d,S", [(torch.float32, 64, 1000), (torch.float16, 64, 1000), (torch.float32, 32, 999),
                                    (torch.bfloat16, 128, 515), (torch.float32, 256, 515)])
def test_edge_tiles_of_every_size(ops, dt, d, S):
    """The first and last tokens of a head are cut into tiles of 16, 32 or 64 by how many heads there are (on 148 SMs and
    S 1000: up to 14 heads, 16, 19): a head's result is the same among any number of heads."""
    most = 19
    g = torch.Generator(device="cuda").manual_seed(S)
    q, k, v = (torch.randn(1, most, S, d, device="cuda", generator=g).to(dt) for _ in range(3))
    pos = torch.randint(0, S, (1, most, S - 6, 3), device="cuda", generator=g, dtype=torch.int32)
    call = lambda n: ops.sparse_attention(*(t[:, :n].contiguous() for t in (q, k, v, pos)), window_size=5, dilation=2,
                                          n_global=3, scale=d ** -0.5)
    whole = call(most)
    for n in (1, 2, 14, 16):
        assert torch.equal(call(n), whole[:, :n])
    ops.check_status()
    ref = dense.sparse_attention_dense(q[0, 0].cpu().double() * d ** -0.5, k[0, 0].cpu().double(), v[0, 0].cpu().double(),
                                       pos[0, 0].cpu(), 5, 2, 3)
    assert (whole[0, 0].cpu().double() - ref).abs().max().item() <= (1e-5 if dt == torch.float32 else 1e-2)


@pytest.mark.parametrize("R", [1, 2, 3, 4])
@pytest.mark.parametrize("dt,d", [(torch.float32, 64), (torch.float16, 64), (torch.bfloat16, 32)])
def test_no_edge_tiles(ops, dt, d, R):
    """A window of one key and no global tokens: every tile is an interior one, a short last one among them."""
    for S in (1, 17, 32, 48, 70, 96, 130, 144, 500):
        for heads in (1, 3):
            q, k, v, pos = _inputs(1, heads, S, d, 0, R, S + heads, dt)
            out = ops.sparse_attention(q.cuda(), k.cuda(), v.cuda(), pos.cuda(), 1, 1, n_global=0)
            ops.check_status()
            ref = dense.sparse_attention_dense(q.double(), k.double(), v.double(), pos, 1, 1, n_global=0)
            # fp32 sums of a few terms of order 1; 16-bit results are rounded once (2^-11, 2^-8)
            assert (out.cpu().double() - ref).abs().max().item() <= {torch.float32: 1e-5, torch.float16: 2e-3, torch.bfloat16: 1e-2}[dt]
