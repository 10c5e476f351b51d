"""The one-kernel layer for very few rows, and the bias in the GEMM's epilogue, against the separate steps, bit for bit."""
from __future__ import annotations

import pytest
import torch

import quest_b200 as quest
from quest_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


# row lengths of one, two and four units of 1024 per warp, with a ragged last unit; rows that fill or exceed the eight warps
@pytest.mark.parametrize("m,k,one_kernel", [(1, 256, True), (4, 1024, True), (4, 4096, True), (2, 5632, True), (3, 5632, False), (1, 11008, True),
                                            (1, 16384, True), (1, 28672, False), (2, 16384, False)])
@pytest.mark.parametrize("block", [64, 128, 256])
def test_one_kernel_layer_equals_quantiser_and_gemm(m, k, one_kernel, block):
    n = 203
    g = torch.Generator(device=DEV).manual_seed(k + m)
    w = (0.02 * torch.randn(n, k, device=DEV, generator=g)).to(torch.bfloat16)
    wp, ws, wa, _ = quest.preprocess_weight(w, use_hadamard=True, block=block)
    x = (torch.randn(m, k, device=DEV, generator=g) * (1 + torch.arange(m, device=DEV))[:, None]).to(torch.bfloat16)
    assert (_lib.load().quest_b200_layer_plan(m, k, n, block) == 2) == one_kernel
    packed, scale, sums = quest.hadamard_quantize_int4(x, block)
    ref = quest.fused_matmul_dequantize_int4_int4t_bf16(packed, wp, sums, wa, scale, ws)
    assert quest.linear_forward(x, wp, ws, wa, use_hadamard=True, block=block).equal(ref)
    zero = torch.zeros_like(x)
    assert quest.linear_forward(zero, wp, ws, wa, use_hadamard=True, block=block).isfinite().all()


# as many weight rows as two blocks per SM hold, and one more
@pytest.mark.parametrize("m", [1, 2])
def test_one_kernel_layer_runs_in_one_round(m):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n, one_kernel in ((64 * sms, True), (64 * sms + 1, False)):
        g = torch.Generator(device=DEV).manual_seed(n)
        w = (0.02 * torch.randn(n, 1024, device=DEV, generator=g)).to(torch.bfloat16)
        wp, ws, wa, _ = quest.preprocess_weight(w, use_hadamard=True)
        x = torch.randn(m, 1024, device=DEV, generator=g).to(torch.bfloat16)
        assert (_lib.load().quest_b200_layer_plan(m, 1024, n, 128) == 2) == one_kernel
        packed, scale, sums = quest.hadamard_quantize_int4(x)
        assert quest.linear_forward(x, wp, ws, wa, use_hadamard=True).equal(quest.fused_matmul_dequantize_int4_int4t_bf16(packed, wp, sums, wa, scale, ws))


@pytest.mark.parametrize("use_hadamard", [True, False])
@pytest.mark.parametrize("m,k,n", [(1, 2048, 96), (12, 2048, 200), (100, 2048, 264), (333, 2048, 1001), (20, 96, 40)])
def test_module_bias(m, k, n, use_hadamard):
    if use_hadamard and k % 128:
        pytest.skip("the transform needs whole blocks")
    torch.manual_seed(m)
    lin = quest.Linear4bit(k, n, bias=True, device=DEV, dtype=torch.bfloat16, use_hadamard=use_hadamard)
    x = torch.randn(m, k, device=DEV).to(torch.bfloat16)
    ref = quest.linear_forward(x, lin.w_int_packed, lin.w_scale, lin.w_add, use_hadamard=use_hadamard)
    ref += lin.bias.detach()
    with torch.inference_mode():
        assert lin(x).equal(ref) and lin(x[None]).equal(ref[None])
    y = lin(x)  # a bias that autograd follows stays an operation of torch
    assert y.equal(ref) and y.requires_grad
    y.float().sum().backward()
    assert lin.bias.grad.float().allclose(torch.full_like(lin.bias, m).float())
