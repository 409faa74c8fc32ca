"""SiLU and its derivative of the whole-network kernels far below zero, where
1 + exp(-z) leaves the range of float32: the value must vanish, however large
-z is (a clamped denominator leaves a multiple of z)."""

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("z", [-80.0, -86.0, -87.0, -87.5, -88.0, -88.5, -89.0, -1e3, -1e30,
                               -1e36, -1e37, -3e38, float("-inf")])
def test_silu_vanishes_far_below_zero(z):
    """h = silu(z) and dz = u silu'(z) against 64 bits.  The float32 formula
    z / (1 + exp(-z)) keeps a relative 1e-4 down to -87 (exp(-z) of a product
    rounded to 2^-24 of its size, 128 log2(e) there) and ends at 0 where
    1 + exp(-z) passes 2^126, at z = -87.34, from a value of 1.03e-36."""
    from pursuit_evasion_b200.learned.mlp import ValueMLP

    rows = 128
    net = ValueMLP(6, layers=1, seed=3, max_batch=rows)
    net.feat.zero_()
    net.target.zero_()
    net.b[0].fill_(z)
    net.loss.zero_()
    net.forward(rows, target=True)
    # the head's gradient is the test's own: y may overflow for infinite h
    net.dy.fill_(1.0)
    net.w_out.fill_(1.0)
    net.backward(rows)
    h, dz = net.h[0].float(), net.dz[0].float()
    if z == float("-inf"):  # -inf / inf, as the formula says
        assert torch.isnan(h).all() and torch.isnan(dz).all()
        return
    v = torch.tensor(z, dtype=torch.float64)
    e = torch.exp(v)
    s = e / (1 + e)
    for got, want in ((h, v * s), (dz, s * (1 + v * (1 - s)))):
        torch.testing.assert_close(got.double(), want.to(net.dev).expand_as(got),
                                   rtol=2.0 ** -7 + 1e-4, atol=1.05e-36)


@pytest.mark.parametrize("z", [-1e3, -3e38])
def test_silu_vanishes_in_a_query(z):
    from pursuit_evasion_b200.learned.mlp import ValueMLP
    from pursuit_evasion_b200.learned.train import predict_states
    from tests.helpers import A3

    net = ValueMLP(6, layers=1, seed=3, max_batch=128)
    net.b[0].fill_(z)
    net.w_out.fill_(1.0)
    net.b_out.fill_(0.25)
    y = predict_states(net, A3, 4.0, torch.zeros(5, 5, device=net.dev))
    assert torch.equal(y, torch.full_like(y, 0.25))
