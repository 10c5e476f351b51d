"""The one-pass scale + quantise kernel (weights behind their transform, activations without one) against the separate
ops it stands for, bit for bit."""
from __future__ import annotations

import pytest
import torch

import quest_b200 as quest

pytestmark = pytest.mark.gpu
DEV = "cuda"


# K around the units of 1024 a warp holds, the longest row, whole 16-byte pieces that are no multiple of 32
@pytest.mark.parametrize("k,block", [(8, 0), (776, 0), (1032, 0), (64, 64), (768, 256), (4096, 128), (5632, 128), (28672, 128), (65536, 256)])
@pytest.mark.parametrize("rows", [1, 37])
def test_one_pass_equals_the_separate_ops(rows, k, block):
    g = torch.Generator(device=DEV).manual_seed(rows + k)
    x = (torch.randn(rows, k, device=DEV, generator=g) * torch.rand(rows, 1, device=DEV, generator=g)).to(torch.bfloat16)
    x[0, : k // 2] = 0
    x[0, : k // 4] = -0.0
    x[rows - 1, k // 2:] *= 1e-6  # quotients far below one, of both signs, beside full-sized ones
    before = x.clone()
    assert quest.one_pass_ok(x, block)
    packed, scale, sums = quest.scale_quantize_int4(x, weight_block=block, row_sum_add=k // 2)
    y = quest.hadamard_transform(x, block=block, weight_side=True) if block else x
    s_ref = quest.find_scale_int4(y)
    p_ref = torch.empty(rows, k // 2, dtype=torch.uint8, device=DEV)
    r_ref = torch.empty(rows, 1, dtype=torch.int32, device=DEV)
    quest.quantize_int4(y, s_ref, x_int_packed=p_ref, x_int_row_sum=r_ref)
    assert packed.equal(p_ref) and scale.equal(s_ref) and sums.equal(r_ref + k // 2) and x.equal(before)


def test_one_pass_refuses_what_it_cannot_hold():
    x = torch.zeros(4, 4096, dtype=torch.bfloat16, device=DEV)
    assert not quest.one_pass_ok(x, 96) and not quest.one_pass_ok(x.float()) and not quest.one_pass_ok(x.t())
    assert not quest.one_pass_ok(torch.zeros(4, 4100, dtype=torch.bfloat16, device=DEV))
    assert not quest.one_pass_ok(torch.zeros(4097, dtype=torch.bfloat16, device=DEV)[1:].view(1, 4096))  # not 16-byte aligned
    w = torch.randn(5, 132, device=DEV).to(torch.bfloat16)  # such a weight takes the separate ops
    packed, scale, add, _ = quest.preprocess_weight(w)
    assert packed.shape == (5, 66) and scale.equal(quest.find_scale_int4(w)) and add.equal(
        (quest.unpack_int4(packed).sum(1, dtype=torch.int32, keepdim=True) + 66))
