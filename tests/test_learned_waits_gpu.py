"""No bounded device wait of the network kernels gives up: every whole-network
pass at small and ragged sizes, then the flag (its raising is tested on the
host; a wait that runs out is never provoked here)."""

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("rows", [128, 9472, 9600])
def test_no_wait_gives_up(rows):
    from pursuit_evasion_b200.learned.mlp import ValueMLP
    from pursuit_evasion_b200.learned.train import RelativeNodeSampler, predict_nodes, predict_states
    from pursuit_evasion_b200.reversible.free_dp import RelativeGrid
    from tests.helpers import A3

    net = ValueMLP(6, seed=3, max_batch=rows)
    net.target.zero_()
    net.loss.zero_()
    net.forward(rows, target=True)
    net.backward(rows)
    net.set_step(1)
    net.adam()
    grid = RelativeGrid(13, 9, 5, 7, 3.0)
    out = predict_nodes(net, RelativeNodeSampler(A3, grid), torch.empty(grid.states, device=net.dev))
    y = predict_states(net, A3, 3.0, torch.zeros(rows - 1, 5, device=net.dev))
    net.check_waits()
    for t in (net.y, net.dy, net.loss, out, y):
        assert torch.isfinite(t).all()
