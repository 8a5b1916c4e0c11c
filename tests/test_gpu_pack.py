"""Parameter packing (csrc/pack.cu) against plain transposes, at sizes that end inside a 64 x 64 tile and rows that do
not begin on 16 bytes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from fractaltensor_b200 import ops as _ops
    return _ops


@pytest.mark.parametrize("dt", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D,I,H", [(1, 64, 64), (3, 128, 192), (2, 24, 40), (1, 7, 5), (2, 65, 129)])
def test_lstm_weights(ops, dt, D, I, H):
    g = torch.Generator(device="cuda").manual_seed(I + H)
    W, U, b = (torch.randn(*s, device="cuda", generator=g).to(dt) for s in ((D, 4, I, H), (D, 4, H, H), (D, 4, H)))
    Wp, bias_p = ops.lstm_pack_weights(W, U, b)
    rows = lambda m: m.permute(0, 3, 1, 2).reshape(D, 4 * H, -1)  # [layer][u * 4 + gate][k]
    assert torch.equal(Wp, torch.cat([rows(W), rows(U)], -1))
    assert torch.equal(bias_p, b.permute(0, 2, 1).reshape(D, 4 * H).float())


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("H,V", [(64, 1), (64, 129), (128, 1000), (512, 997), (64, 256)])
def test_projection(ops, dt, H, V):
    P = torch.randn(H, V, device="cuda").to(dt)
    Pt = ops.projection_pack(P)
    assert torch.equal(Pt[:V], P.t()) and Pt[V:].eq(0).all()


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H", [64, 72, 128])
def test_grid_and_rnn_weights(ops, dt, H):
    a, b = torch.randn(2, 2 * H, H, device="cuda").to(dt), torch.randn(2, H, H, device="cuda").to(dt)
    assert torch.equal(ops.grid_pack_weights(a, b), torch.cat([a, b], 1).transpose(1, 2))
    W, U = torch.randn(H + 8, H, device="cuda").to(dt), torch.randn(H, H, device="cuda").to(dt)
    assert torch.equal(ops.rnn_pack_weights(W, U), torch.cat([W, U], 0).t())
