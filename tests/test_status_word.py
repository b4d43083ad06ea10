"""The kernels' status word and those who look at it, on the host alone: a sampler whose kernels are stood in for, and a word that
tells when it is cleared."""
import pytest
import torch

from geneinfer_b200 import SamplingParams
from geneinfer_b200.ops import kernels
from geneinfer_b200.sampling.device import DeviceSampler


class Word:
    """The word [1], calling ``cleared`` at the moment when it no longer holds a failure."""

    def __init__(self):
        self.value, self.cleared = 0, lambda: None

    def __getitem__(self, i):
        return self.value

    def __setitem__(self, i, value):
        was, self.value = self.value, int(value)
        if was and not self.value:
            self.cleared()

    def zero_(self):
        self[0] = 0


class Event:
    def record(self):
        pass

    def synchronize(self):
        pass


class Host:
    """A sampler of two tokens on the host; ``sample()`` is a call under way, ``launched`` runs where its kernels are launched."""

    def __init__(self):
        self.device = torch.device("cpu", 0)
        self.state = kernels._tc_states[0]
        self.sampler = DeviceSampler(2, self.device)
        self.launched = lambda: None

    def argmax(self, logits, ids):
        self.launched()
        ids.copy_(logits.argmax(1))

    def sample(self):
        return self.sampler.sample_async(torch.tensor([[0.0, 1.0]]), [SamplingParams(0.0)], [0.0])


@pytest.fixture
def host(monkeypatch):
    monkeypatch.setattr(torch.Tensor, "pin_memory", lambda self, *a: self)
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)
    state = kernels._TensorCoreState(torch.device("cpu", 0))
    state.status = Word()
    monkeypatch.setitem(kernels._tc_states, 0, state)
    h = Host()
    monkeypatch.setattr(kernels, "argmax", h.argmax)
    return h


def test_a_failure_is_counted_before_the_word_is_cleared(host):
    """Another thread that looks at the very moment when the word is cleared still learns of the failure."""
    one, other = host.sample(), host.sample()
    seen = []

    def look():
        with pytest.raises(kernels.KernelError):
            other.result()
        seen.append(True)

    host.state.status[0] = 0x21
    host.state.status.cleared = look
    with pytest.raises(kernels.KernelError, match="0x21"):
        one.result()
    assert seen == [True] and host.sample().result() == [1]


def test_a_failure_while_a_sample_is_launched_is_its_own(host):
    """Another thread finds and clears a failure between the launch of a sample's kernels and the end of the call that launches them."""
    def fail():
        host.state.status[0] = 0x22
        assert kernels.take_failure(host.device, kernels.status_failures(host.device))

    host.launched = fail
    call = host.sample()
    host.launched = lambda: None
    with pytest.raises(kernels.KernelError):
        call.result()
    assert host.sample().result() == [1]


def test_a_failure_ends_when_its_kernels_have(host, monkeypatch):
    """A kernel that has given up one wait gives up others while it runs on: they belong to the same failure, and a call that is made
    after it has been raised is not ended by them."""
    running = [True]

    def ends():
        if running.pop() and not host.state.status[0]:
            host.state.status[0] = 0x23
        running.append(False)

    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: ends())
    call = host.sample()
    host.state.status[0] = 0x21
    with pytest.raises(kernels.KernelError):
        call.result()
    ends()
    assert host.sample().result() == [1]


def test_every_call_under_way_names_the_failure(host):
    """Who learns of a failure by the count gives its code too."""
    calls = [host.sample(), host.sample()]
    host.state.status[0] = 0x21
    for call in calls:
        with pytest.raises(kernels.KernelError, match="status 0x21"):
            call.result()
