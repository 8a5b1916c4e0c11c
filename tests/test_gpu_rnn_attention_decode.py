"""The attention RNN whose decoder is one launch behind the encoder's scan (csrc/rnn_attention.cu, attn_decode_kernel) against the
three launches that calls without its scratch take, from the C entry: odd numbers of sequences, steps and positions around the
sizes a warp requests ahead, every cluster size, sequences without positions, and terms that are not finite."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _call(src, trg, q, lens, whole):
    from fractaltensor_b200 import ops
    from fractaltensor_b200.ops import _dtype_code, _ptr, _stream, check, lib
    (Ls, N, H), Lt = src.shape, trg.shape[0]
    buf = lambda *s, dt=src.dtype: torch.full(s, 7.0, dtype=dt, device="cuda")
    enc, scores, dec, out = buf(Ls, N, H), buf(Ls, N, dt=torch.float32), buf(Lt, N, H), buf(Lt, N, H)
    code = _dtype_code(src)
    encoder, everything = lib.ftb_rnn_attention_scratch_bytes(Ls, N, H, code), lib.ftb_rnn_attention_scratch_bytes_all(Ls, Lt, N, H, code)
    assert everything == encoder + Lt * N * H * 4  # (all calls here have the one launch)
    scratch = torch.full((everything if whole else encoder,), 255, dtype=torch.uint8, device="cuda")
    ws = ops.workspace(src.device)
    check(lib.ftb_rnn_attention_fwd_scratch(_ptr(src), _ptr(trg), _ptr(q["Wp_src"]), _ptr(q["Wp_trg"]), _ptr(q["bs"]), _ptr(q["bt"]),
                                            _ptr(q["enc_proj"]), _ptr(q["dec_proj"]), _ptr(lens) if lens is not None else None,
                                            _ptr(enc), _ptr(scores), _ptr(dec), _ptr(out), Ls, Lt, N, H, code, _ptr(scratch),
                                            scratch.numel(), _ptr(ws), ws.numel(), _stream()), "ftb_rnn_attention_fwd_scratch")
    ops.check_status()
    return enc, scores, dec, out


def _inputs(dt, H, Ls, Lt, N):
    from fractaltensor_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(H + Ls + Lt + N)
    uni = lambda *s: (torch.rand(*s, device="cuda", generator=g) * 2 - 1) / math.sqrt(H)
    q = {k: ops.rnn_pack_weights(uni(H, H).to(dt), uni(H, H).to(dt)) for k in ("Wp_src", "Wp_trg")}
    q.update(bs=uni(H), bt=uni(H))
    # (a projection may begin anywhere: one does, one not, on a 16-byte boundary)
    q["enc_proj"], q["dec_proj"] = torch.rand(H, device="cuda", generator=g).to(dt), torch.rand(H + 1, device="cuda", generator=g).to(dt)[1:]
    src, trg = (torch.randn(n, N, H, device="cuda", generator=g).to(dt) for n in (Ls, Lt))
    return src, trg, q


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("H,Ls,Lt,N,lens", [
    (128, 1, 1, 1, None), (256, 5, 9, 3, [5, 0, 2]), (384, 64, 64, 2, [64, 63]), (512, 65, 65, 5, [65, 1, 33, 0, 64]),
    (512, 256, 128, 4, [256, 255, 31, 128]), (128, 130, 8, 33, None), (256, 17, 63, 72, None), (512, 12, 30, 72, None),
])
def test_as_the_three_launches(dt, H, Ls, Lt, N, lens):
    src, trg, q = _inputs(dt, H, Ls, Lt, N)
    lens = None if lens is None else torch.tensor(lens, dtype=torch.int32, device="cuda")
    one, three = _call(src, trg, q, lens, True), _call(src, trg, q, lens, False)
    assert torch.equal(one[0], three[0]) and torch.equal(one[1], three[1])
    # states and vectors are sums in another order, rounded to 16 bits: one unit in the last place of numbers up to 1
    ulp = 2.0 ** -11 if dt == torch.float16 else 2.0 ** -8
    for a, b in zip(one[2:], three[2:]):
        assert (a.float() - b.float()).abs().max().item() <= ulp
        assert (a != b).float().mean().item() <= 0.02


@pytest.mark.parametrize("H,N", [(128, 3), (512, 4)])
def test_what_is_not_finite(H, N):
    Ls, Lt = 6, 70
    src, trg, q = _inputs(torch.bfloat16, H, Ls, Lt, N)
    lens = torch.tensor([6, 0, 3, 5][:N], dtype=torch.int32, device="cuda")
    for at in (0, 7, 8, 63, 64, Lt - 1):
        bad = trg.clone()
        bad[at, 0, H - 1] = float("nan")
        bad[at, 1, 3] = float("nan")  # a sequence that attends to nothing
        one, three = _call(src, bad, q, lens, True), _call(src, bad, q, lens, False)
        for a, b in zip(one[2:], three[2:]):
            assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.isnan(one[3][at:, 0]).all() and not torch.isnan(one[3][:at]).any()
            assert (a.float() - b.float()).nan_to_num().abs().max().item() <= 2.0 ** -8


def test_in_a_graph_and_behind_one_another():
    """Dependent launches in a row, each reading what the one before wrote, as a graph too."""
    from fractaltensor_b200 import ops
    src, trg, q = _inputs(torch.bfloat16, 256, 9, 20, 16)
    args = (q["Wp_src"], q["Wp_trg"], q["bs"], q["bt"], q["enc_proj"], q["dec_proj"])

    def links():
        x = trg
        for _ in range(4):
            x = ops.rnn_attention(src, x, *args)[1]
        return x

    want = links().clone()
    torch.cuda.synchronize()
    for _ in range(3):
        assert torch.equal(links(), want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = links()
    for _ in range(2):
        got.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)
    ops.check_status()
