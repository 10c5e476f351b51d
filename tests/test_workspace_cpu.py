"""The activation workspaces a module keeps: what stays cached, and the packed form where memory does not hold the int8 operand."""
from __future__ import annotations

import pytest
import torch

from quest_b200 import workspace
from quest_b200.workspace import KEPT_OPERAND, WorkspaceCache, layer_workspaces

DEVICE = torch.device("cuda", 0)


@pytest.fixture
def allocations(monkeypatch):
    """Stand-ins for device memory; a size in ``full`` does not fit."""
    class Record(list):
        full = ()

    made = Record()

    def empty(*shape, dtype=None, device=None):
        if shape in made.full:
            raise torch.OutOfMemoryError(f"{shape}")
        made.append(shape)
        return torch.zeros(1, dtype=dtype).expand(shape)

    monkeypatch.setattr(workspace.torch, "empty", empty)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: 0, raising=False)
    return made


def test_a_set_is_kept_up_to_the_size_of_an_operand(allocations):
    cache = WorkspaceCache()
    k = 4096
    m = KEPT_OPERAND // k
    assert cache.get(m, k, DEVICE, int8_operand=True) is cache.get(m, k, DEVICE, int8_operand=True)
    assert cache.get(m + 1, k, DEVICE, int8_operand=True) is not cache.get(m + 1, k, DEVICE, int8_operand=True)
    assert cache.get(4 * m, k, DEVICE) is cache.get(4 * m, k, DEVICE)
    assert cache.nbytes() == KEPT_OPERAND + 6 * m + 2 * KEPT_OPERAND + 24 * m


def test_a_layer_falls_back_to_packed_codes(allocations):
    cache = WorkspaceCache()
    allocations.full = ((64, 512),)
    ws = layer_workspaces(cache, 64, 512, DEVICE, torch.bfloat16, True)
    assert "_a_int8" not in ws and ws["_a_int_packed"].shape == (64, 256)
    allocations.full = ()
    assert layer_workspaces(cache, 64, 512, DEVICE, torch.bfloat16, True)["_a_int8"].shape == (64, 512)
    allocations.full = ((64, 1024), (64, 512))
    with pytest.raises(torch.OutOfMemoryError):
        layer_workspaces(cache, 64, 1024, DEVICE, torch.bfloat16, True)
