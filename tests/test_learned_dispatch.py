"""Which inference route predict_nodes and predict_states take: the one-launch
kernels stand for the package's own features and network only, a subclass that
overrides `encode` or `forward` is asked (host logic, no GPU needed)."""

from types import SimpleNamespace

import pytest

torch = pytest.importorskip("torch")

from pursuit_evasion_b200.learned import train
from pursuit_evasion_b200.learned.mlp import FEATURES, ValueMLP
from pursuit_evasion_b200.reversible.free_dp import RelativeGrid
from tests.helpers import A3

GRID = RelativeGrid(5, 4, 3, 3, 2.0)


def host_net(cls, rows=256):
    """The attributes of a network that inference reads, in host memory."""
    net = cls.__new__(cls)
    net.torch, net.dev, net.hidden, net.layers, net.batch = torch, torch.device("cpu"), 256, 4, rows
    net.feat = torch.zeros(rows, FEATURES)
    net.y = torch.zeros(rows)
    return net


class FirstFeature(ValueMLP):
    """The first feature is the value."""

    def forward(self, rows, *, target=False, inference=False):
        self.y[:rows] = self.feat[:rows, 0]
        return self.y[:rows]


class OwnFeatures(train.RelativeNodeSampler):
    def encode(self, net, idx, rows, with_target):
        net.feat[:rows, 0] = 3.0 * idx[:rows].float()


@pytest.fixture
def one_launch(monkeypatch):
    """Replace the one-launch routes by records of their calls."""
    calls = []

    def predict(self, net, first, rows, out):
        calls.append(rows)
        out.copy_(torch.arange(first, first + rows))

    monkeypatch.setattr(train.RelativeNodeSampler, "predict", predict)
    return calls


def test_overridden_encode_is_asked(one_launch):
    net = host_net(FirstFeature)
    sampler = OwnFeatures(A3, GRID)
    out = train.predict_nodes(net, sampler, torch.empty(GRID.states))
    assert torch.equal(out, 3.0 * torch.arange(GRID.states, dtype=torch.float32))
    assert not one_launch


def test_overridden_encode_is_asked_with_the_packages_network(one_launch, monkeypatch):
    net = host_net(ValueMLP)
    monkeypatch.setattr(ValueMLP, "forward", FirstFeature.forward)
    out = train.predict_nodes(net, OwnFeatures(A3, GRID), torch.empty(GRID.states))
    assert torch.equal(out, 3.0 * torch.arange(GRID.states, dtype=torch.float32))
    assert not one_launch


def test_encode_of_an_instance_is_asked(one_launch, monkeypatch):
    net = host_net(ValueMLP)
    monkeypatch.setattr(ValueMLP, "forward", FirstFeature.forward)
    sampler = train.RelativeNodeSampler(A3, GRID)
    sampler.encode = lambda net, idx, rows, with_target: OwnFeatures.encode(
        sampler, net, idx, rows, with_target)
    out = train.predict_nodes(net, sampler, torch.empty(GRID.states))
    assert torch.equal(out, 3.0 * torch.arange(GRID.states, dtype=torch.float32))
    assert not one_launch


def test_overridden_forward_is_asked(one_launch, monkeypatch):
    net = host_net(FirstFeature)
    sampler = train.RelativeNodeSampler(A3, GRID)
    monkeypatch.setattr(train.RelativeNodeSampler, "encode", OwnFeatures.encode)
    out = train.predict_nodes(net, sampler, torch.empty(GRID.states))
    assert torch.equal(out, 3.0 * torch.arange(GRID.states, dtype=torch.float32))
    assert not one_launch


def test_a_sampler_and_network_of_another_kind(one_launch):
    """Anything with the attributes that the loop reads, as before there was a
    one-launch route."""
    sampler = SimpleNamespace(cells=300, encode=lambda net, idx, rows, t: OwnFeatures.encode(
        None, net, idx, rows, t), predict=None)
    net = SimpleNamespace(**vars(host_net(FirstFeature)))
    net.forward = lambda rows, inference: FirstFeature.forward(net, rows)
    out = train.predict_nodes(net, sampler, torch.empty(300))
    assert torch.equal(out, 3.0 * torch.arange(300, dtype=torch.float32))


def test_the_packages_own_take_one_launch(one_launch):
    net = host_net(ValueMLP)
    out = train.predict_nodes(net, train.RelativeNodeSampler(A3, GRID), torch.empty(GRID.states))
    assert torch.equal(out, torch.arange(GRID.states, dtype=torch.float32))


def test_overridden_forward_is_asked_by_queries(monkeypatch):
    def unused(*args):
        raise AssertionError("the one-launch route was taken")

    def encode(states, n, *args):
        net.feat[:n, 0] = 7.0
        return 0

    monkeypatch.setattr(train._native, "library", lambda: SimpleNamespace(
        pe_mlp_encode_relative_states=encode, pe_mlp_predict_relative_states=unused))
    net = host_net(FirstFeature)
    net._stream = lambda: None
    net.native_net = unused
    got = train.predict_states(net, A3, 2.0, torch.zeros(3, 5))
    assert torch.equal(got, torch.full((3,), 7.0))


@pytest.mark.parametrize("out", ["double", "strided"])
def test_results_of_another_layout_go_through_a_bounded_buffer(monkeypatch, out):
    """A destination that the kernel cannot write directly costs a buffer of at
    most 32 MB, not one of the whole table."""
    n = (1 << 23) + 1001
    pieces = []

    def predict(self, net, first, rows, values):
        assert values.dtype == torch.float32 and values.is_contiguous() and values.numel() == rows
        pieces.append((first, rows))
        values.copy_(torch.arange(first, first + rows))

    monkeypatch.setattr(train.RelativeNodeSampler, "predict", predict)
    sampler = train.RelativeNodeSampler(A3, GRID)
    sampler.cells = n
    table = (torch.zeros(n + 3, dtype=torch.float64) if out == "double"
             else torch.zeros(n + 3, 2)[:, 1])
    assert train.predict_nodes(host_net(ValueMLP), sampler, table) is table
    assert torch.equal(table[:n], torch.arange(n, dtype=table.dtype))
    assert not table[n:].any()
    assert max(4 * rows for _, rows in pieces) <= 32 << 20
