"""The whole-network kernels (csrc/mlp_fused.cu) against the launch-per-layer
kernels on the same weights: activations, outputs and gradients at the
smallest and ragged row counts and at one, four and eight layers; bulk and
online inference at ragged sizes; SiLU at extreme pre-activations."""

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

BF16_ULP = 2.0 ** -7  # of the value, at most


def make_net(layers, rows, seed=3, in_features=6):
    from pursuit_evasion_b200.learned.mlp import ValueMLP

    net = ValueMLP(in_features, layers=layers, seed=seed, max_batch=rows)
    g = torch.Generator().manual_seed(seed + 1)
    net.feat.zero_()
    net.feat[:, :in_features] = torch.randn(rows, in_features, generator=g).to(net.dev)
    net.target.copy_(torch.randn(rows, generator=g))
    return net


def per_layer(net):
    """The same network on the launch-per-layer kernels."""
    cls = type("PerLayer", (type(net),), {"fused": property(lambda self: False)})
    net.__class__ = cls
    return net


def step(net, rows):
    net.loss.zero_()
    y = net.forward(rows, target=True).clone()
    net.backward(rows)
    net.set_step(1)
    grads = [g.clone() for g in net.grads]
    out = dict(y=y, loss=net.loss.clone(), z=[t.clone() for t in net.z],
               h=[t.clone() for t in net.h], dz=[t.clone() for t in net.dz], grads=grads)
    torch.cuda.synchronize()
    return out


def close_norm(a, b, rel):
    d = (a.double() - b.double()).norm()
    assert float(d) <= rel * float(b.double().norm()) + 1e-30


@pytest.mark.parametrize("layers,rows", [(1, 128), (4, 128), (4, 384), (4, 2048), (8, 256)])
def test_fused_step_equals_the_per_layer_kernels(layers, rows):
    net = make_net(layers, rows)
    assert net.fused
    new = step(net, rows)
    old = step(per_layer(net), rows)
    # the same MMA sequence: pre-activations differ only where an activation
    # before them rounded to the other side of a bf16 boundary
    assert torch.equal(new["z"][0], old["z"][0])
    for name in ("h", "dz"):
        for a, b in zip(new[name], old[name]):
            torch.testing.assert_close(a.float(), b.float(), rtol=BF16_ULP, atol=1e-7)
            assert float((a != b).float().mean()) < 1e-3
    torch.testing.assert_close(new["y"], old["y"], rtol=1e-5, atol=1e-6)
    torch.testing.assert_close(new["loss"], old["loss"], rtol=1e-5, atol=0)
    # FP32 sums of `rows` terms in another order
    for a, b in zip(new["grads"], old["grads"]):
        close_norm(a, b, 1e-4)


def test_fused_adam_equals_the_per_layer_kernels():
    rows = 128
    a, b = make_net(4, rows), make_net(4, rows)
    for net in (a, per_layer(b)):
        for g, p in zip(net.grads, net.params):
            g.copy_(torch.sin(37.0 * p) * 0.1)
        net.set_step(3)
        net.adam(lr=1e-2)
    for x, y in zip(a.params + a.m + a.v + a.w16 + a.w16t, b.params + b.m + b.v + b.w16 + b.w16t):
        assert torch.equal(x, y)


@pytest.mark.parametrize("n", [1, 127, 129, 1000, 148 * 128 + 1, 40001])
def test_fused_query_equals_the_per_layer_kernels(n):
    from pursuit_evasion_b200.learned.train import predict_states
    from tests.helpers import A3

    net = make_net(4, (n + 127) // 128 * 128)
    g = torch.Generator().manual_seed(n)
    states = ((torch.rand(n, 5, generator=g) * 2 - 1) * 4).to(net.dev)
    new = predict_states(net, A3, 4.0, states)
    old = predict_states(per_layer(net), A3, 4.0, states)
    assert new.shape == (n,)
    torch.testing.assert_close(new, old, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("world", [False, True])
def test_fused_nodes_equal_the_per_layer_kernels(world):
    from pursuit_evasion_b200.learned import train
    from pursuit_evasion_b200.reversible.free_dp import RelativeGrid
    from pursuit_evasion_b200.reversible.world_dp import WorldGrid
    from tests.helpers import A3

    if world:
        sampler = train.WorldNodeSampler(A3, WorldGrid(5, 5, 4, 3, 3.0))
    else:
        sampler = train.RelativeNodeSampler(A3, RelativeGrid(13, 9, 5, 7, 3.0))
    net = make_net(4, 4096, in_features=sampler.in_features)
    n = sampler.cells
    new = train.predict_nodes(net, sampler, torch.empty(n, device=net.dev))
    strided = torch.zeros(n, 2, device=net.dev)[:, 0]  # not contiguous
    train.predict_nodes(net, sampler, strided)
    assert torch.equal(strided, new)
    old = train.predict_nodes(per_layer(net), sampler, torch.empty(n, device=net.dev))
    torch.testing.assert_close(new, old, rtol=1e-5, atol=1e-6)


def test_silu_at_extreme_pre_activations():
    rows = 128
    net = make_net(1, rows)
    for z in (0.0, -0.5, 20.0, -20.0, -80.0, -87.0, -120.0, 300.0, float("inf"), float("nan")):
        net.feat.zero_()
        net.b[0].fill_(z)
        net.loss.zero_()
        net.forward(rows, target=True)
        net.backward(rows)
        h, dz = net.h[0].float(), net.dz[0].float()
        v = torch.tensor(z, dtype=torch.float64)
        want = v / (1 + torch.exp(-v))
        if torch.isfinite(want):
            torch.testing.assert_close(h, torch.full_like(h, float(want)), rtol=BF16_ULP,
                                       atol=1e-30)
            assert torch.isfinite(dz).all()
        else:
            assert torch.equal(torch.isnan(h), torch.full_like(h, float(want)).isnan())
            assert not torch.isfinite(h).any()


@pytest.mark.parametrize("layers", [1, 2, 4])
def test_two_ctas_per_tile_equal_one(layers):
    """A forward training pass shares a 128-row tile between two CTAs up to 74
    tiles (9472 rows) and gives it to one from 75: the same rows either way, and
    their backward pass."""
    many, few = 9600, 9472
    net = make_net(layers, many)
    runs = []
    for rows in (many, few):
        net.loss.zero_()
        net.forward(rows, target=True)
        # the mean's 1 / rows is the one difference between the two calls
        net.dy.copy_((net.y - net.target) * (2.0 / many))
        net.backward(rows)
        torch.cuda.synchronize()
        runs.append([t[:few].clone() for t in [net.y] + net.z + net.h + net.dz])
    for a, b in zip(*runs):
        assert torch.equal(a, b)
    # FP32 sums of the second run: at most 608 roundings of 2^-24 (chains of 16
    # rows, 8 ranges and 74 tiles) on the sum of magnitudes
    bound = 608 * 2.0 ** -24
    pairs = [(net.grads[layers + l], net.dz[l][:few].double()) for l in range(layers)]
    dy = net.dy[:few].double()[:, None]
    pairs.append((net.grads[2 * layers], dy * net.h[-1][:few].double()))
    pairs.append((net.grads[2 * layers + 1], dy))
    for got, terms in pairs:
        err = (got.double().flatten() - terms.sum(0)).abs()
        assert bool((err <= bound * terms.abs().sum(0) + 1e-30).all())
