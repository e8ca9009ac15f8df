"""When a solver asks for the larger scratch area: any that is small beside the card, larger ones only where as much again
stays free."""
import types

import pytest
import torch


@pytest.mark.parametrize("area,free,held,share,fits", [
    (8, 0, 0, 1.0, True),  # small beside the card: the allocation itself will tell
    (20, 39, 0, 1.0, False),
    (20, 40, 0, 1.0, True),
    (20, 30, 10, 1.0, True),  # what the allocator holds and nobody uses counts as free
    (20, 150, 0, 0.25, False),  # of 40 that the process may use, 2 are in use
    (20, 150, 0, 0.3, True),
])
def test_room_for_the_larger_area(monkeypatch, area, free, held, share, fits):
    from poker2_b200 import solver

    gib = 1 << 30
    for name, value in {"get_device_properties": types.SimpleNamespace(total_memory=160 * gib), "memory_allocated": 2 * gib,
                        "memory_reserved": (2 + held) * gib, "get_per_process_memory_fraction": share,
                        "mem_get_info": (free * gib, 160 * gib)}.items():
        monkeypatch.setattr(torch.cuda, name, lambda device, value=value: value)
    assert solver._room_for(area * gib, torch.device("cuda:0")) == fits
