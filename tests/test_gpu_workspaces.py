"""Workspaces of the caller in ``linear_forward``: any subset, larger ones, both code buffers; the same bits and the same route as
without, and the checks that buffers of other shapes meet."""
from __future__ import annotations

import itertools

import pytest
import torch

import quest_b200 as quest
from quest_b200.workspace import WorkspaceCache

pytestmark = pytest.mark.gpu
DEV = "cuda"


def layer(m, k, n, use_hadamard=True):
    g = torch.Generator(device=DEV).manual_seed(m + k + n)
    w = (0.02 * torch.randn(n, k, device=DEV, generator=g)).to(torch.bfloat16)
    wp, ws, wa, _ = quest.preprocess_weight(w, use_hadamard=use_hadamard)
    return torch.randn(m, k, device=DEV, generator=g).to(torch.bfloat16), wp, ws, wa


def buffers(m, k, rows=None):
    return {"_a_int8": torch.zeros(m, k, dtype=torch.uint8, device=DEV), "_a_int_packed": torch.zeros(m, k // 2, dtype=torch.uint8, device=DEV),
            "_a_scale": torch.zeros(rows or m, 1, dtype=torch.bfloat16, device=DEV),
            "_a_int_row_sum": torch.zeros(rows or m, 1, dtype=torch.int32, device=DEV)}


# one token (the one-kernel form has no workspaces to fill), the few-token kernel, a K that only the mma.sync quantiser tiles, a K
# without an int8 operand
@pytest.mark.parametrize("m,k,n", [(1, 512, 96), (40, 5632, 200), (300, 2048, 264), (9, 192, 40)])
@pytest.mark.parametrize("use_hadamard", [True, False])
def test_any_subset_of_workspaces(m, k, n, use_hadamard):
    if use_hadamard and k % 128:
        pytest.skip("the transform needs whole blocks")
    x, wp, ws, wa = layer(m, k, n, use_hadamard)
    ref = quest.linear_forward(x, wp, ws, wa, use_hadamard=use_hadamard)
    for rows in (None, m + 5):
        for names in itertools.chain.from_iterable(itertools.combinations(("_a_int8", "_a_int_packed", "_a_scale", "_a_int_row_sum"), r) for r in range(1, 5)):
            given = {name: t for name, t in buffers(m, k, rows).items() if name in names}
            assert quest.linear_forward(x, wp, ws, wa, use_hadamard=use_hadamard, **given).equal(ref), names
            for name in ("_a_scale", "_a_int_row_sum"):
                if name in given:
                    assert given[name][:m].count_nonzero() > 0 and given[name][m:].count_nonzero() == 0
            codes = [name for name in ("_a_int8", "_a_int_packed") if name in given]
            if len(codes) == 2:  # the buffer of the library's own choice
                codes = ["_a_int8"] if quest.layer_operand(m, k, n) else ["_a_int_packed"]
            for name in ("_a_int8", "_a_int_packed"):
                if name in given and k % 128 == 0:
                    assert (given[name].count_nonzero() > 0) == (name in codes), names


def test_buffers_of_other_shapes_are_still_refused():
    m, k, n = 40, 512, 96
    x, wp, ws, wa = layer(m, k, n)
    for use_hadamard in (True, False):
        with pytest.raises(AssertionError):  # a weight of another K
            quest.linear_forward(x, wp[:, :128].contiguous(), ws, wa, use_hadamard=use_hadamard)
        with pytest.raises(AssertionError):
            quest.linear_forward(x, wp, ws, wa, use_hadamard=use_hadamard, out=torch.empty(n, m, dtype=torch.bfloat16, device=DEV).t())
        both = buffers(m, k)
        with pytest.raises(AssertionError):  # a batch of matrices
            quest.linear_forward(x.view(4, 10, k), wp, ws, wa, use_hadamard=use_hadamard, **both)
    with pytest.raises(AssertionError):
        quest.linear_forward(x, wp, ws, wa, use_hadamard=True, out=torch.empty(m, n + 8, dtype=torch.bfloat16, device=DEV))
    assert quest.linear_forward(x[:0], wp, ws, wa, use_hadamard=True).shape == (0, n)


@pytest.mark.parametrize("module", [False, True])
def test_a_layer_fits_where_its_packed_form_does(module):
    """With room for the output and the packed codes only: the allocator's own limit stands in for a full device."""
    m, k, n = 32768, 8192, 1536
    x, wp, ws, wa = layer(m, k, n)
    lin = quest.Linear4bit(k, n, bias=False, device=DEV, dtype=torch.bfloat16, use_hadamard=True)
    lin.w_int_packed, lin.w_scale, lin.w_add = wp, ws, wa
    lin.workspaces = WorkspaceCache()
    call = (lambda: lin(x)) if module else (lambda: quest.linear_forward(x, wp, ws, wa, use_hadamard=True))
    assert quest.layer_operand(m, k, n)
    with torch.inference_mode():
        ref = call()
        lin.workspaces.clear()
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        room = 2 * m * n + m * k // 2 + (64 << 20)  # less than half of the int8 operand's second half to spare
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + room) / torch.cuda.get_device_properties(0).total_memory)
        try:
            y = call()
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0)
    # the packed route may quantise with another kernel, which may round a transform output the other way
    assert (y.float() - ref.float()).norm() <= 1e-2 * ref.float().norm()
    assert not module or {"_a_int_packed"} == {name for ws_ in lin.workspaces._sets.values() for name in ws_ if name.startswith("_a_int") and name != "_a_int_row_sum"}
