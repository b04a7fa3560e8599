"""The library of host code that reads PyTorch tensors: what it takes as an expert slot, and which build of it is loaded."""
import ctypes
import types

import pytest
import torch


def addresses(slots, n=None):
    from macseek_b200 import _lib, quant
    out = (ctypes.c_uint64 * (3 * max(len(slots), 1)))(*([7] * (3 * max(len(slots), 1))))
    _lib.host().msb_slot_addresses(slots, quant.ExpertSlot, len(slots) if n is None else n, out)
    return list(out)[:3 * len(slots)]


class Lazy:
    gate = property(lambda self: None)
    up = down = None


def test_slots_of_any_class():
    from macseek_b200.quant import ExpertSlot

    class Sub(ExpertSlot):
        pass

    assert addresses([ExpertSlot(), types.SimpleNamespace(gate=None, up=None, down=None), Lazy(), Sub()]) == [0] * 12
    assert addresses((ExpertSlot(),)) == [0] * 3 and addresses([]) == []
    with pytest.raises(AttributeError):
        addresses([types.SimpleNamespace(gate=None, up=None)])
    with pytest.raises(AssertionError):                       # not on the device
        addresses([ExpertSlot(gate=torch.zeros(1))])
    with pytest.raises(AssertionError):
        addresses([types.SimpleNamespace(gate=None, up=torch.zeros(1), down=None)])
    with pytest.raises(IndexError):
        addresses([ExpertSlot(), ExpertSlot()], 1)


def test_a_slot_takes_attributes_of_its_user():
    from macseek_b200.quant import ExpertSlot
    s = ExpertSlot(1, 2, 3)
    s.layer = 5
    s.up = 4
    assert (s.gate, s.up, s.down, s.layer) == (1, 4, 3, 5)


def test_a_library_for_another_pytorch_is_rebuilt_and_not_loaded(monkeypatch):
    from macseek_b200 import _lib, build
    _lib.host()
    assert build._host_target() == _lib.host_target() and not build._host_stale(build._host_target())
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    assert build._host_stale(build._host_target())
    with pytest.raises(ImportError, match="0.0.1"):
        _lib.host.__wrapped__()


@pytest.mark.gpu
def test_addresses_are_the_tensors():
    from macseek_b200.quant import ExpertSlot
    t = [torch.zeros(8, device="cuda")[k:] for k in range(3)]
    want = [v.data_ptr() for v in t]
    assert addresses([ExpertSlot(*t), types.SimpleNamespace(gate=t[0], up=t[1], down=t[2]), ExpertSlot(up=t[1])]) == 2 * want + [0, want[1], 0]
