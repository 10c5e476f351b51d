"""What the fused decoder block keeps of autograd, on the CPU with stand-ins for the kernels (which know no graph): the residual
path of a block carries gradients and forward-mode tangents to its input, as the sums of torch that it replaces do."""
from __future__ import annotations

import pytest
import torch
import torch.autograd.forward_ad as fwAD
from torch import nn

import quest_b200 as quest
from quest_b200 import prefill
from quest_b200.prefill import Block, DecoderConfig, RMSNorm, apply_rope, rope_table


class Quantised(nn.Module):
    """A linear as the block sees it: whatever goes in, its output has no graph."""

    def __init__(self, k, n):
        super().__init__()
        self.in_features, self.out_features = k, n
        self.register_buffer("w", 0.05 * torch.randn(n, k))

    def forward_quantized(self, codes, scale, sums):
        return (codes.detach().float() @ self.w.T).to(torch.bfloat16)

    def forward(self, x):
        return self.forward_quantized(x, None, None)


@pytest.fixture
def block(monkeypatch):
    torch.manual_seed(0)
    cfg = DecoderConfig(n_embd=32, n_layer=1, n_head=2, ffn=64)
    blk = Block(cfg).to(torch.bfloat16)
    blk.attn.c_attn, blk.attn.c_proj = Quantised(32, 96), Quantised(32, 32)
    blk.mlp.w1, blk.mlp.w2, blk.mlp.c_proj = Quantised(32, 64), Quantised(32, 64), Quantised(64, 32)
    blk.fused = True

    def raw(t):  # what a kernel sees: memory
        return fwAD.unpack_dual(t).primal.detach() if fwAD._current_level >= 0 else t.detach()

    def norm(x, w, eps):
        xf = x.float()
        return (xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps)).to(x.dtype) * w

    def produce(kind, x, codes=None, scale=None, x_int_row_sum=None, x2=None, norm_weight=None, eps=0.0, block=128):
        y = norm(raw(x), raw(norm_weight), eps) if kind == quest.PRODUCE_RMSNORM else nn.functional.silu(raw(x)) * raw(x2)
        return y, scale, x_int_row_sum

    def add_produce(x, y, norm_weight, eps, block=128, **outputs):
        total = raw(x) + raw(y)
        return total, produce(quest.PRODUCE_RMSNORM, total, norm_weight=norm_weight, eps=eps)

    def rope(x, table, seq, cols):
        with torch.no_grad():
            q, k = (raw(x)[:, i * cols // 2:(i + 1) * cols // 2].view(-1, seq, blk.attn.n_head, cols // 2 // blk.attn.n_head) for i in (0, 1))
            q2, k2 = apply_rope(q, k, table)
            q.copy_(q2), k.copy_(k2)

    monkeypatch.setattr(quest, "producer_hadamard_quantize", produce)
    monkeypatch.setattr(quest, "add_rmsnorm_hadamard_quantize", add_produce)
    monkeypatch.setattr(quest, "rope_inplace", rope)
    monkeypatch.setattr(quest, "layer_operand", lambda *a: False)
    monkeypatch.setattr(prefill.default_cache, "get", lambda *a, **k: {"_a_int_packed": None, "_a_scale": None, "_a_int_row_sum": None})
    return blk


def test_the_residual_carries_the_gradient(block):
    table = rope_table(16, 8)
    x = torch.randn(1, 8, 32).to(torch.bfloat16).requires_grad_()
    with torch.no_grad():
        ref = block(x, table)
    y = block(x, table)
    assert y.equal(ref) and y.requires_grad
    g = torch.randn(1, 8, 32).to(torch.bfloat16)
    y.backward(g)
    assert x.grad.equal(g)  # both sums are the identity in x, everything else has no graph


def test_the_residual_carries_a_tangent(block):
    table = rope_table(16, 8)
    x, t = (torch.randn(1, 8, 32).to(torch.bfloat16) for _ in range(2))
    with torch.no_grad(), fwAD.dual_level():
        y, tangent = fwAD.unpack_dual(block(fwAD.make_dual(x, t), table))
    assert y.equal(block(x, table)) and tangent is not None and tangent.equal(t)


class OnDevice(torch.Tensor):
    """A CPU tensor that says it is on the GPU, to see which form the norm takes."""
    is_cuda = True


def test_the_norm_keeps_its_eager_form_where_the_kernel_cannot_follow(monkeypatch):
    calls = []
    monkeypatch.setattr(quest, "rmsnorm", lambda x, w, eps: calls.append(1) or x)
    norm = RMSNorm(16, 1e-5).to(torch.bfloat16)
    norm.fused = True
    x = torch.randn(3, 16).to(torch.bfloat16).as_subclass(OnDevice)
    with torch.no_grad():
        norm(x)
        assert len(calls) == 1
        with fwAD.dual_level():
            norm(x)
        assert len(calls) == 1
        norm.weight = nn.Parameter(torch.ones(32).to(torch.bfloat16)[::2])  # strided
        norm(x)
        norm.weight = nn.Parameter(torch.ones(1).to(torch.bfloat16))  # broadcast
        norm(x)
    assert len(calls) == 1
