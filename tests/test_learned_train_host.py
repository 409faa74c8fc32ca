"""Host side of the training loop (no GPU needed): what it orders between
streams, with stand-ins for the streams that record it."""

from contextlib import contextmanager
from types import SimpleNamespace

import pytest

torch = pytest.importorskip("torch")

from pursuit_evasion_b200.learned import train


class Streams:
    """torch with a recorder in the place of torch.cuda."""

    def __init__(self):
        self.log = []
        self.caller = self.current = self.Stream()
        self.log.clear()
        self.cuda = self

    def __getattr__(self, name):
        return getattr(torch, name)

    def Stream(self, device=None):
        s = SimpleNamespace()
        s.wait_stream = lambda other: self.log.append(("wait", s, other))
        return s

    def current_stream(self, device=None):
        return self.current

    @contextmanager
    def stream(self, s):
        before, self.current = self.current, s
        yield
        self.current = before

    def synchronize(self, device=None):
        self.log.append(("synchronize",))


def host_net(streams):
    net = SimpleNamespace(torch=streams, dev=torch.device("cpu"), batch=64,
                          loss=torch.zeros(1), set_step=lambda step: None)
    for name in ("forward", "backward", "adam"):
        setattr(net, name, lambda *args, **kwargs: None)
    net.check_waits = lambda: streams.log.append(("check",))
    return net


def test_training_waits_for_what_the_caller_queued():
    """Parameters, table and sample list belong to the caller's stream: the
    loop's own stream waits for it before the first sample is read."""
    streams = Streams()
    net = host_net(streams)

    def encode(net, idx, rows, with_target):
        streams.log.append(("read", streams.current))

    sampler = SimpleNamespace(cells=100, encode=encode)
    train.train(net, sampler, samples=64, epochs=1, batch=64, use_graph=False)
    reads = [e for e in streams.log if e[0] == "read"]
    assert len(reads) == 1 and reads[0][1] is not streams.caller
    wait = ("wait", reads[0][1], streams.caller)
    assert wait in streams.log
    assert streams.log.index(wait) < streams.log.index(reads[0])


def test_training_checks_the_device_waits_at_its_end():
    streams = Streams()
    net = host_net(streams)
    sampler = SimpleNamespace(cells=100, encode=lambda *args: streams.log.append(("read",)))
    train.train(net, sampler, samples=128, epochs=2, batch=64, use_graph=False)
    assert streams.log[-1] == ("check",) and streams.log.count(("read",)) == 4


@pytest.mark.parametrize("gave_up", [0, 1])
def test_a_wait_that_gave_up_is_raised(gave_up):
    from pursuit_evasion_b200 import _native
    from pursuit_evasion_b200.learned.mlp import ValueMLP

    def timeouts(count):
        count._obj.value = gave_up
        return 0

    streams = Streams()
    net = ValueMLP.__new__(ValueMLP)
    net.torch, net.dev = streams, torch.device("cpu")
    net.lib = SimpleNamespace(pe_mlp_gemm_tc_timeouts=timeouts)
    if gave_up:
        with pytest.raises(_native.NativeError, match="gave up"):
            net.check_waits()
    else:
        net.check_waits()
    assert streams.log == [("synchronize",)]
