"""CPU: training stops when a kernel of a step did not finish.  The library is a
fake whose error flag is set by the host; the network does no work."""
import ctypes

import pytest

from alamo_gb300 import AgbError, learned


class FakeLib:
    def __init__(self, fail_at):
        self.calls, self.fail_at = 0, fail_at

    def agb_conv3_tc_error(self, flag):
        self.calls += 1
        flag._obj.value = int(self.calls == self.fail_at)
        return 0

    def agb_last_error(self):
        return b""


class FakeNet:
    def __init__(self):
        self.steps = 0

    def forward(self, g0, feat):
        import torch
        return torch.ones((g0[0] ** 3, learned.FEAT), requires_grad=False)

    def backward(self, g0, dout):
        return [], []

    def adam(self, gw, gb, lr):
        self.steps += 1


def samples(n):
    import torch
    return [{"feat": None, "target": torch.rand((n + 1) ** 3, 3) + 0.5}]


def test_training_runs_without_the_flag(monkeypatch):
    fake, net = FakeLib(0), FakeNet()
    monkeypatch.setattr(learned, "lib", lambda: fake)
    assert len(learned.train(net, samples(2), 2, steps=4)) == 4
    assert net.steps == 4 and fake.calls == 5


@pytest.mark.parametrize("at", [1, 3, 5])
def test_training_stops_on_the_flag(monkeypatch, at):
    fake, net = FakeLib(at), FakeNet()
    monkeypatch.setattr(learned, "lib", lambda: fake)
    with pytest.raises(AgbError):
        learned.train(net, samples(2), 2, steps=4)
    assert net.steps == at - 1
    flag = ctypes.c_int(1)
    fake.agb_conv3_tc_error(ctypes.byref(flag))
    assert flag.value == 0
