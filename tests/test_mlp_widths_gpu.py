"""Networks of other widths than 256, which run a launch per layer: gradients
against FP64 autograd on the same bf16 weights, inference of nodes and states
against the forward pass, and a training run."""

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

BF16_ULP = 2.0 ** -7  # of the value, at most


def bf16(t):
    return t.to(torch.bfloat16).double()


class RoundGrad(torch.autograd.Function):
    """Identity forward; the incoming gradient rounded to bf16 (the kernels
    store activation gradients in it)."""

    @staticmethod
    def forward(ctx, t):
        return t.clone()

    @staticmethod
    def backward(ctx, grad):
        return bf16(grad)


def make_net(hidden, layers, rows):
    from pursuit_evasion_b200.learned.mlp import ValueMLP

    net = ValueMLP(6, hidden=hidden, layers=layers, seed=3, max_batch=rows)
    assert not net.fused
    return net


@pytest.mark.parametrize("hidden,layers,rows", [(128, 1, 128), (128, 4, 640), (384, 3, 256),
                                                (512, 2, 384)])
def test_gradients_of_other_widths_match_fp64_autograd(hidden, layers, rows):
    """As at width 256: what is left is FP32 against FP64 accumulation and the
    rare value that rounds to the other side of a bf16 boundary, so every
    gradient agrees within half a bf16 unit in the last place, in norm."""
    net = make_net(hidden, layers, rows)
    g = torch.Generator().manual_seed(1)
    feat = torch.zeros(rows, net.feat.shape[1])
    feat[:, :6] = torch.rand(rows, 6, generator=g) * 2 - 1
    target = torch.sin(3 * feat[:, 0]) * feat[:, 1] + 0.5 * feat[:, 4]
    net.feat.copy_(feat.to(torch.bfloat16))
    net.target.copy_(target)
    net.loss.zero_()
    y = net.forward(rows, target=True)
    net.backward(rows)
    net.check_waits()

    ws = [w.double().cpu().requires_grad_() for w in net.w16]
    bs = [b.double().cpu().requires_grad_() for b in net.b]
    wo = net.w_out.double().cpu().requires_grad_()
    bo = net.b_out.double().cpu().requires_grad_()
    h = net.feat.double().cpu()
    for w, b in zip(ws, bs):
        z = RoundGrad.apply(h @ w.t() + b)
        h = torch.nn.functional.silu(z)
        h = h + (bf16(h) - h).detach()
    ref = h @ wo + bo
    loss = ((ref - target.double()) ** 2).mean()
    loss.backward()
    torch.testing.assert_close(y.double().cpu(), ref.detach(), rtol=0.5 * BF16_ULP, atol=1e-3)
    assert float(net.loss) == pytest.approx(loss.item(), rel=1e-3)
    for ours, want in zip(net.grads, [t.grad for t in ws + bs + [wo, bo]]):
        ours = ours.double().cpu().reshape(want.shape)
        assert float((ours - want).norm()) < 0.5 * BF16_ULP * max(float(want.norm()), 1e-12)


@pytest.mark.parametrize("hidden", [128, 384])
def test_inference_and_training_of_other_widths(hidden):
    from pursuit_evasion_b200.learned import train
    from pursuit_evasion_b200.reversible.free_dp import RelativeGrid
    from tests.helpers import A3

    grid = RelativeGrid(13, 9, 5, 7, 3.0)
    net = make_net(hidden, 3, 512)
    sampler = train.RelativeNodeSampler(A3, grid)
    out = train.predict_nodes(net, sampler, torch.empty(grid.states, device=net.dev), chunk=512)
    axes = grid.axes(A3)
    cells = torch.arange(0, grid.states, 97)[:300]
    iv, ie, ip, iy, ix = torch.unravel_index(cells, grid.shape)
    pick = lambda a, i: torch.tensor(a, dtype=torch.float32)[i]
    states = torch.stack([pick(axes[4], ix), pick(axes[3], iy), pick(axes[2], ip),
                          pick(axes[0], iv), pick(axes[1], ie)], 1).to(net.dev)
    got = train.predict_states(net, A3, grid.extent, states)
    # one state as node and as query: its features may round to neighbouring bf16
    torch.testing.assert_close(got, out[cells.to(net.dev)], rtol=0, atol=2e-2)
    sampler.table = torch.sin(out * 3.0) + 0.5
    losses, _ = train.train(net, sampler, samples=1 << 13, epochs=6, batch=512)
    assert losses[-1] < 0.5 * losses[0]
