"""Entries that make room for others (``DeviceLedger.on_pressure``)."""
import pytest
import torch

from owl_engine_b200.utils.ledger import BudgetError, DeviceLedger


def test_a_convenience_makes_room_and_a_need_is_still_refused():
    led = DeviceLedger("cpu", total_bytes=1000, enforce=True)
    held = [led.alloc("convenience", "workspace", (600,), torch.uint8)]
    calls = []

    def give_back():
        calls.append(1)
        if held:
            held.clear()
            led.release("convenience")
    led.on_pressure(give_back)
    led.on_pressure(give_back)
    led.alloc("small", "workspace", (300,), torch.uint8)
    assert not calls                                    # it fitted beside it
    led.alloc("large", "workspace", (600,), torch.uint8)
    assert calls == [1] and sorted(led.entries) == ["large", "small"]
    with pytest.raises(BudgetError):
        led.alloc("too large", "workspace", (200,), torch.uint8)
    assert led.refused == 1
