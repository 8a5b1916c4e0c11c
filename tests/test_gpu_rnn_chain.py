"""The encoder scan of the attention RNN as one launch (csrc/rnn_chain.cu): slices of 16 sequences, 128
units a CTA, a scan cut into pieces, against one launch per position and fp64."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(ops, lib, x, y, Wp, bias, proj, pieces):
    """ftb_rnn_attention_fwd with room for `pieces` steps of the input half (0: one launch per position)."""
    Ls, N, H = x.shape
    enc, dec, out = torch.empty_like(x), torch.empty_like(y), torch.empty_like(y)
    scores = torch.empty(Ls, N, device="cuda")
    ws = torch.zeros(lib.ftb_workspace_bytes() + pieces * N * H * 4, dtype=torch.uint8, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    rc = lib.ftb_rnn_attention_fwd(p(x), p(y), p(Wp), p(Wp), p(bias), p(bias), p(proj), p(proj), None, p(enc),
                                   p(scores), p(dec), p(out), Ls, y.shape[0], N, H, ops._dtype_code(x), p(ws),
                                   ws.numel(), ops._stream())
    assert rc == 0
    torch.cuda.synchronize()
    assert int(ws[:4].view(torch.int32)) == 0
    return enc, out


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("H,N,Ls", [
    (64, 1, 5),      # half a tile of units, one sequence
    (128, 16, 2),    # one full CTA, one full slice, the shortest scan with a hand-off
    (192, 17, 9),    # a full and a half tile, a slice of one sequence
    (512, 33, 7),    # the widest: four CTAs
    (384, 16, 1),    # no hand-off at all
])
def test_chain_matches_levels_and_fp64(dt, H, N, Ls):
    from fractaltensor_b200 import ops
    from fractaltensor_b200._lib import lib
    g = torch.Generator(device="cuda").manual_seed(H + N)
    u = lambda *s: ((torch.rand(*s, device="cuda", generator=g) * 2 - 1) / H ** 0.5).to(dt)
    W, U, bias, proj = u(H, H), u(H, H), u(H).float(), u(H)
    x, y = (torch.randn(n, N, H, device="cuda", generator=g).to(dt) for n in (Ls, 3))
    Wp = ops.rnn_pack_weights(W, U)
    levels, _ = _run(ops, lib, x, y, Wp, bias, proj, 0)
    whole, out = _run(ops, lib, x, y, Wp, bias, proj, Ls)
    cut, out_cut = _run(ops, lib, x, y, Wp, bias, proj, 2)
    assert torch.equal(whole, cut) and torch.equal(out, out_cut)  # the pieces hand the state on exactly
    # One rounding to the stored type per step: |h| <= 1, so half a unit in the last place is at most
    # 2^-12 (fp16) or 2^-9 (bf16); an error of a state reaches the next through U (row sums at most
    # sqrt(H) / 2 in expectation 1/2 of that) with tanh' <= 1, and tanh.approx adds 2^-11: four such units.
    tol = 4 * (2.0 ** -11 + (2.0 ** -12 if dt == torch.float16 else 2.0 ** -9))
    h = torch.zeros(N, H, dtype=torch.float64, device="cuda")
    for t in range(Ls):
        h = torch.tanh(x[t].double() @ W.double() + h @ U.double() + bias.double())
        assert (whole[t].double() - h).abs().max().item() <= tol
        assert (levels[t].double() - h).abs().max().item() <= tol


@pytest.mark.parametrize("H", [64, 192, 320, 448])  # odd multiples of 64: half of the last CTA's warps have no units
def test_long_scans_with_warps_without_units(H):
    """Those warps take no part in the steps: a scan of many steps ends with status 0 and the states of the
    level launches' arithmetic."""
    from fractaltensor_b200 import ops
    from fractaltensor_b200._lib import lib
    N, Ls, dt = 40, 400, torch.float16
    g = torch.Generator(device="cuda").manual_seed(H)
    u = lambda *s: ((torch.rand(*s, device="cuda", generator=g) * 2 - 1) / H ** 0.5).to(dt)
    W, U, bias, proj = u(H, H), u(H, H), u(H).float(), u(H)
    x, y = (torch.randn(n, N, H, device="cuda", generator=g).to(dt) for n in (Ls, 2))
    Wp = ops.rnn_pack_weights(W, U)
    tol = 4 * (2.0 ** -11 + 2.0 ** -12)  # as above
    for _ in range(5):
        enc, _out = _run(ops, lib, x, y, Wp, bias, proj, Ls)
    h = torch.zeros(N, H, dtype=torch.float64, device="cuda")
    for t in range(Ls):
        h = torch.tanh(x[t].double() @ W.double() + h @ U.double() + bias.double())
        assert (enc[t].double() - h).abs().max().item() <= tol


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("H,N,Ls", [(64, 16, 6), (192, 17, 9), (320, 5, 3), (512, 33, 40), (256, 3, 1), (384, 50, 2)])
def test_chain_has_the_bits_of_the_level_launches(dt, H, N, Ls):
    """The scan adds the state's products to the input half in the order of the cell kernel, so that a call's
    result does not depend on how much scratch it had, whole or in pieces of any length."""
    from fractaltensor_b200 import ops
    from fractaltensor_b200._lib import lib
    g = torch.Generator(device="cuda").manual_seed(H + Ls)
    u = lambda *s: ((torch.rand(*s, device="cuda", generator=g) * 2 - 1) / H ** 0.5).to(dt)
    x, y = (torch.randn(n, N, H, device="cuda", generator=g).to(dt) for n in (Ls, 3))
    Wp, bias, proj = ops.rnn_pack_weights(u(H, H), u(H, H)), u(H).float(), u(H)
    levels, out = _run(ops, lib, x, y, Wp, bias, proj, 0)
    for pieces in sorted({1, 2, 3, Ls}):
        enc, o = _run(ops, lib, x, y, Wp, bias, proj, min(pieces, Ls))
        assert torch.equal(enc, levels) and torch.equal(o, out)
