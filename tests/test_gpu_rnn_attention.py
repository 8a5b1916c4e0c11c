"""GPU parity of the attention RNN (examples/rnn_attention/rnn_attention.py:40-110) with the oracle
and with the fixture the reference's frontend produced."""
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


def _ragged(flat, lens):
    from fractaltensor_b200 import frontend
    return frontend.FractalTensor(flat.cuda(), [list(range(int(n))) for n in lens], (1, flat.shape[1]))


def _params(H, seed, bound):
    g = torch.Generator().manual_seed(seed)
    uni = lambda *s: (torch.rand(*s, generator=g) * 2 - 1) * bound
    return dict(Ws=uni(H, H), Us=uni(H, H), bs=uni(1, H), Wt=uni(H, H), Ut=uni(H, H), bt=uni(1, H),
                enc_proj=torch.rand(H, 1, generator=g), dec_proj=torch.rand(H, 1, generator=g)), g


def test_rnn_attention_golden(ops, golden_dir):
    """The reference frontend's own result on ragged batches (H = 16 there; the kernels take multiples
    of 64, so the fixture's parameters are embedded in H = 64 with zeros, which leaves the first 16
    columns of every state unchanged)."""
    from fractaltensor_b200 import frontend
    g = _load(golden_dir, "rnn_attention_small.npz")
    h, H = g["src"].shape[1], 64
    pad_m = lambda m: torch.nn.functional.pad(m, (0, H - m.shape[1], 0, H - m.shape[0]))
    pad_r = lambda m: torch.nn.functional.pad(m, (0, H - m.shape[1]))
    pad_c = lambda m: torch.nn.functional.pad(m, (0, 0, 0, H - m.shape[0]))
    # padded units: zero weights and zero bias -> tanh(0) = 0 everywhere, and zero projection rows
    src, trg = _ragged(pad_r(g["src"]), g["src_lens"]), _ragged(pad_r(g["trg"]), g["trg_lens"])
    out = frontend.rnn_attention(src, trg, (pad_m(g["Ws"]).cuda(), pad_m(g["Us"]).cuda(), pad_r(g["bs"]).cuda()),
                                 (pad_m(g["Wt"]).cuda(), pad_m(g["Ut"]).cuda(), pad_r(g["bt"]).cuda()),
                                 (pad_c(g["enc_proj"]).cuda(), pad_c(g["dec_proj"]).cuda()))
    ops.check_status()
    assert [len(i) for i in out.indices] == g["trg_lens"].tolist() and out.element_shape == (1, H)
    got = out.data.reshape(-1, H).cpu()
    assert (got[:, :h] - g["out"]).abs().max().item() <= 1e-5
    assert got[:, h:].abs().max().item() == 0


@pytest.mark.parametrize("dt", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("H,src_lens,trg_lens", [
    (64, [5, 3, 7], [4, 6, 2]),
    (128, [9] * 4, [5] * 4),                       # rectangular
    (256, list(range(1, 41)), list(range(40, 0, -1))),  # 40 sequences, lengths 1..40
    (512, [30, 17, 50, 50, 2, 41, 8], [20, 33, 5, 12, 40, 1, 9]),  # the example's hidden size and batch
])
def test_rnn_attention_matches_oracle(ops, dt, H, src_lens, trg_lens):
    from fractaltensor_b200 import frontend
    p, g = _params(H, H + len(src_lens), 1.0 / (H ** 0.5))
    src = torch.randn(sum(src_lens), H, generator=g).to(dt)
    trg = torch.randn(sum(trg_lens), H, generator=g).to(dt)
    pq = {k: v.to(dt) for k, v in p.items()}
    out = frontend.rnn_attention(_ragged(src, src_lens), _ragged(trg, trg_lens),
                                 (pq["Ws"].cuda(), pq["Us"].cuda(), pq["bs"].cuda()),
                                 (pq["Wt"].cuda(), pq["Ut"].cuda(), pq["bt"].cuda()),
                                 (pq["enc_proj"].cuda(), pq["dec_proj"].cuda()))
    ops.check_status()
    d64 = {k: v.double() for k, v in pq.items()}
    _, ref = dense.rnn_attention_dense(src.double(), trg.double(), src_lens, trg_lens, d64["Ws"], d64["Us"], d64["bs"],
                                       d64["Wt"], d64["Ut"], d64["bt"], d64["enc_proj"], d64["dec_proj"])
    got = out.data.reshape(-1, H).cpu().double()
    err = (got - ref).abs().max().item()
    if dt == torch.float32:
        assert err <= 1e-5 * max(1.0, ref.abs().max().item()), err
    else:
        assert err <= 2e-2, err


def test_rnn_attention_dense_entry(ops):
    """The tensor-level entry on a rectangular time-major batch without lengths, encoder states included."""
    H, Ls, Lt, N = 128, 12, 7, 130
    p, g = _params(H, 5, 1.0 / (H ** 0.5))
    dt = torch.bfloat16
    src, trg = torch.randn(Ls, N, H, generator=g).to(dt), torch.randn(Lt, N, H, generator=g).to(dt)
    pq = {k: v.to(dt) for k, v in p.items()}
    enc, out = ops.rnn_attention(src.cuda(), trg.cuda(), ops.rnn_pack_weights(pq["Ws"].cuda(), pq["Us"].cuda()),
                                 ops.rnn_pack_weights(pq["Wt"].cuda(), pq["Ut"].cuda()),
                                 pq["bs"].reshape(H).float().cuda(), pq["bt"].reshape(H).float().cuda(),
                                 pq["enc_proj"].reshape(H).cuda(), pq["dec_proj"].reshape(H).cuda())
    ops.check_status()
    d64 = {k: v.double() for k, v in pq.items()}
    for n in (0, 64, 129):
        e_ref, o_ref = dense.rnn_attention_dense(src[:, n].double(), trg[:, n].double(), [Ls], [Lt], d64["Ws"], d64["Us"],
                                                 d64["bs"], d64["Wt"], d64["Ut"], d64["bt"], d64["enc_proj"],
                                                 d64["dec_proj"])
        assert (enc[:, n].cpu().double() - e_ref).abs().max().item() <= 2e-2
        assert (out[:, n].cpu().double() - o_ref).abs().max().item() <= 2e-2


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_rnn_attention_smallest_shapes(ops, dt):
    """One sequence, one source and one target position; and a batch that is not a multiple of any tile."""
    from fractaltensor_b200 import frontend
    for src_lens, trg_lens in (([1], [1]), ([1, 2, 1], [2, 1, 3])):
        H = 64
        p, g = _params(H, 3 + len(src_lens), 1.0 / (H ** 0.5))
        src = torch.randn(sum(src_lens), H, generator=g).to(dt)
        trg = torch.randn(sum(trg_lens), H, generator=g).to(dt)
        pq = {k: v.to(dt) for k, v in p.items()}
        out = frontend.rnn_attention(_ragged(src, src_lens), _ragged(trg, trg_lens),
                                     (pq["Ws"].cuda(), pq["Us"].cuda(), pq["bs"].cuda()),
                                     (pq["Wt"].cuda(), pq["Ut"].cuda(), pq["bt"].cuda()),
                                     (pq["enc_proj"].cuda(), pq["dec_proj"].cuda()))
        ops.check_status()
        d64 = {k: v.double() for k, v in pq.items()}
        _, ref = dense.rnn_attention_dense(src.double(), trg.double(), src_lens, trg_lens, d64["Ws"], d64["Us"],
                                           d64["bs"], d64["Wt"], d64["Ut"], d64["bt"], d64["enc_proj"], d64["dec_proj"])
        err = (out.data.reshape(-1, H).cpu().double() - ref).abs().max().item()
        assert err <= (1e-5 if dt == torch.float32 else 2e-2), err
        # with a single source position the attention vector is that encoder state, whatever the scores
        if src_lens == [1]:
            enc1 = torch.tanh(src.double() @ d64["Ws"] + d64["bs"])
            assert (out.data.reshape(-1, H).cpu().double() - enc1).abs().max().item() <= (1e-5 if dt == torch.float32 else 2e-2)


@pytest.mark.parametrize("dt", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("Lt", [2, 40])
def test_what_is_not_finite_reaches_the_later_steps(ops, dt, Lt):
    """A decoder state that is not finite makes its step's weights NaN, and by the recurrent input every later
    step of that sequence; the others and the steps before keep their values."""
    Ls, N, H = 7, 9, 64
    p, g = _params(H, 5, 1.0 / 8)
    q = {k: v.to(dt).cuda() for k, v in p.items()}
    src, trg = (torch.randn(n, N, H, generator=g).to(dt).cuda() for n in (Ls, Lt))
    lens = torch.tensor([7, 3, 5, 7, 1, 2, 6, 0, 4], dtype=torch.int32, device="cuda")
    clean = trg.clone()
    trg[0, 1, 3] = float("nan")            # from the first step on
    trg[Lt - 1, 2, 0] = float("nan")       # the last step alone
    trg[Lt // 2, 4, :2] = float("inf")     # inf - inf in some units, where their weights differ in sign
    trg[Lt // 2, 7, 5] = float("nan")      # a sequence that attends to nothing
    src[2, 5, 0] = float("nan")            # past that sequence's length
    call = lambda t: ops.rnn_attention(src, t, ops.rnn_pack_weights(q["Ws"], q["Us"]),
                                       ops.rnn_pack_weights(q["Wt"], q["Ut"]), q["bs"].float().reshape(-1),
                                       q["bt"].float().reshape(-1), q["enc_proj"].reshape(-1), q["dec_proj"].reshape(-1),
                                       lens)[1]
    out, finite = call(trg), call(clean)
    ops.check_status()
    d = {k: v.double() for k, v in q.items()}
    h, enc = torch.zeros(N, H, dtype=torch.float64, device="cuda"), []
    for t in range(Ls):
        h = torch.tanh(src[t].double() @ d["Ws"] + h @ d["Us"] + d["bs"])
        enc.append(h)
    enc = torch.stack(enc)
    keys = (torch.arange(Ls, device="cuda")[:, None] < lens[None]).unsqueeze(-1)
    enc = torch.where(keys, enc, torch.zeros_like(enc))
    s0 = torch.where(keys[..., 0], (enc @ d["enc_proj"])[..., 0], torch.full((Ls, N), -np.inf, device="cuda").double())
    v, bad = torch.zeros(N, H, dtype=torch.float64, device="cuda"), []
    for t in range(Lt):
        dec = torch.tanh(trg[t].double() @ d["Wt"] + v @ d["Ut"] + d["bt"])
        w = torch.softmax(s0 + (dec @ d["dec_proj"])[:, 0], 0)
        v = (torch.where(keys, w.unsqueeze(-1) * enc, torch.zeros_like(enc))).sum(0)
        bad.append(torch.isnan(v))
    bad = torch.stack(bad)
    assert torch.equal(torch.isnan(out), bad) and bad.any() and not bad.all()
    assert torch.equal(out[~bad], finite[~bad])


@pytest.mark.parametrize("dt", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("H,Ls,Lt,lens", [
    (64, 300, 3, [300, 1, 77, 0]),       # more source positions than threads; nothing to attend to
    (192, 5, 70, [5, 3, 4]),             # more target steps than row groups; columns that end inside a CTA's 128
    (640, 9, 2, [9, 8, 2, 1, 5]),        # wider than the scan kernel takes
])
def test_vectors_of_all_steps(ops, dt, H, Ls, Lt, lens):
    """One attention vector a sequence in the rows of all its steps, scores and sums in one launch."""
    N = len(lens)
    p, g = _params(H, H + Ls, 1.0 / (H ** 0.5))
    src, trg = torch.randn(Ls, N, H, generator=g).to(dt), torch.randn(Lt, N, H, generator=g).to(dt)
    pq = {k: v.to(dt) for k, v in p.items()}
    enc, out = ops.rnn_attention(src.cuda(), trg.cuda(), ops.rnn_pack_weights(pq["Ws"].cuda(), pq["Us"].cuda()),
                                 ops.rnn_pack_weights(pq["Wt"].cuda(), pq["Ut"].cuda()),
                                 pq["bs"].reshape(H).float().cuda(), pq["bt"].reshape(H).float().cuda(),
                                 pq["enc_proj"].reshape(H).cuda(), pq["dec_proj"].reshape(H).cuda(),
                                 torch.tensor(lens, dtype=torch.int32).cuda())
    ops.check_status()
    for n, m in enumerate(lens):
        if m == 0:
            assert out[:, n].eq(0).all()
            continue
        e = enc[:m, n].double().cpu()
        w = torch.softmax(e @ pq["enc_proj"].double().reshape(H), 0)
        ref = (w @ e).expand(Lt, H)  # the decoder's term moves all scores alike
        # fp32 scores of H products (relative 2^-24 * sqrt(H)) in the exponent, then the rounding of the result
        tol = {torch.float32: 1e-5, torch.float16: 1e-3, torch.bfloat16: 8e-3}[dt]
        assert (out[:, n].double().cpu() - ref).abs().max().item() <= tol


def _whole(ops, src, trg, q, lens=None):
    """The C entry itself -> (enc, scores, dec, out), from buffers of sevens."""
    from fractaltensor_b200.ops import _dtype_code, _ptr, _stream, check, lib
    (Ls, N, H), Lt = src.shape, trg.shape[0]
    buf = lambda *s, dt=src.dtype: torch.full(s, 7.0, dtype=dt, device="cuda")
    enc, scores, dec, out = buf(Ls, N, H), buf(Ls, N, dt=torch.float32), buf(Lt, N, H), buf(Lt, N, H)
    bs, bt = (q[k].float().reshape(-1) for k in ("bs", "bt"))
    Wp_src, Wp_trg = ops.rnn_pack_weights(q["Ws"], q["Us"]), ops.rnn_pack_weights(q["Wt"], q["Ut"])
    ws = ops.workspace(src.device)
    check(lib.ftb_rnn_attention_fwd_scratch(_ptr(src), _ptr(trg), _ptr(Wp_src), _ptr(Wp_trg), _ptr(bs), _ptr(bt),
                                            _ptr(q["enc_proj"]), _ptr(q["dec_proj"]), _ptr(lens), _ptr(enc), _ptr(scores),
                                            _ptr(dec), _ptr(out), Ls, Lt, N, H, _dtype_code(src), None, 0, _ptr(ws),
                                            ws.numel(), _stream()), "ftb_rnn_attention_fwd_scratch")
    ops.check_status()
    return enc, scores, dec, out


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,Lt", [(1, 33), (2, 700), (1, 5000)])
def test_steps_shared_by_several_ctas(ops, dt, N, Lt):
    """A step that is not finite reaches the later ones where other CTAs look at those."""
    p, g = _params(64, N + Lt, 1.0 / 8)
    q = {k: v.to(dt).cuda() for k, v in p.items()}
    src, trg = (torch.randn(n, N, 64, generator=g).to(dt).cuda() for n in (5, Lt))
    clean = _whole(ops, src, trg, q)
    assert all(torch.isfinite(t).all() for t in clean)
    for first in (0, 31, 32, Lt - 1):
        trg_bad = trg.clone()
        trg_bad[first, 0, 3] = float("nan")
        if first + 40 < Lt:
            trg_bad[first + 40, 0, 0] = float("nan")  # and one behind it
        _, _, dec, out = _whole(ops, src, trg_bad, q)
        for got, ref in ((dec, clean[2]), (out, clean[3])):
            assert torch.isnan(got[first:, 0]).all()
            assert torch.equal(got[:first], ref[:first]) and torch.equal(got[:, 1:], ref[:, 1:])


@pytest.mark.parametrize("dt", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("H,Ls,lens", [(64, 5, None), (64, 5, [5, 0, 3]), (192, 70, [1, 70, 33, 34, 69])])
def test_scores_of_all_positions(ops, dt, H, Ls, lens):
    """enc_scores holds e_j . enc_proj of every row of enc, past a sequence's length too."""
    N = 2 if lens is None else len(lens)
    p, g = _params(H, H + Ls, 1.0 / (H ** 0.5))
    q = {k: v.to(dt).cuda() for k, v in p.items()}
    src, trg = (torch.randn(n, N, H, generator=g).to(dt).cuda() for n in (Ls, 3))
    enc, scores, _, _ = _whole(ops, src, trg, q, None if lens is None else torch.tensor(lens, dtype=torch.int32).cuda())
    ref = (enc.double() @ q["enc_proj"].double())[..., 0]
    # fp32 sums of H products of at most 1
    assert (scores.double() - ref).abs().max().item() <= H * 2.0 ** -23
