"""What ChunkFeeder refuses before a kernel is launched (no GPU: the library is a stub that must not be reached)."""
import pytest
import torch

from mathbrain_b200 import _lib, feeder as feeder_module
from mathbrain_b200.feeder import ChunkFeeder


class Unreachable:
    def __getattr__(self, name):
        raise AssertionError("library call %s reached" % name)


@pytest.fixture
def feeder(monkeypatch):
    """A feeder of two documents whose resident tensors are on `meta`, standing for one GPU; `cpu` stands for another."""
    monkeypatch.setattr(feeder_module, "_require_cuda", lambda *t: None)
    monkeypatch.setattr(feeder_module._lib, "load", lambda: Unreachable())
    return ChunkFeeder(2, 50, torch.ones(4), capacity=8, device="meta")


def operands():
    return dict(x=torch.zeros(2, 6, dtype=torch.long, device="meta"), fill=torch.zeros(2, dtype=torch.int32, device="meta"),
                C_seq=torch.zeros(2, 6, 4, device="meta"))


@pytest.mark.parametrize("name", ["x", "fill", "C_seq"])
def test_operands_of_another_device(feeder, name):
    ops = operands()
    ops[name] = torch.zeros_like(ops[name], device="cpu")
    with pytest.raises(_lib.MbemaError, match="operand on cpu"):
        feeder.advance(ops["x"], ops["fill"], ops["C_seq"])
    if name != "C_seq":
        with pytest.raises(_lib.MbemaError, match="operand on cpu"):
            feeder.next_batch(ops["x"], ops["fill"])


@pytest.mark.parametrize("name", ["last_t", "seen", "n_seen", "t0", "rhos"])
def test_resident_tensors_of_another_device_or_shape(feeder, name):
    ops = operands()
    for other in (torch.zeros_like(getattr(feeder, name), device="cpu"), getattr(feeder, name)[:1]):
        held = getattr(feeder, name)
        setattr(feeder, name, other)
        with pytest.raises(_lib.MbemaError, match=name):
            feeder.advance(ops["x"], ops["fill"], ops["C_seq"])
        setattr(feeder, name, held)


def test_changed_lists_are_checked_on_the_device(feeder):
    """The widest list that next_batch read bounds the lists after the chunk only while they are the ones it was read from."""
    def after(change):
        feeder._widest = 3, feeder._lists()
        change()
        return feeder._longest_possible(4)
    assert after(lambda: None) == 7 and feeder._widest is None
    assert feeder._longest_possible(4) > feeder.cap                        # no next_batch before
    for change in (lambda: feeder.n_seen.fill_(6), lambda: feeder.seen.zero_(), lambda: feeder.reset([0]),
                   lambda: setattr(feeder, "n_seen", feeder.n_seen.clone()), lambda: setattr(feeder, "seen", feeder.seen.clone())):
        assert after(change) > feeder.cap
