"""What the fused decoder block adds to the quantisers: the in-place rotary embedding and the residual add in front of the
norm, against their eager forms, bit for bit."""
from __future__ import annotations

import pytest
import torch

import quest_b200 as quest
from quest_b200.prefill import Decoder, DecoderConfig, apply_rope, rope_in_place_ok, rope_table, swap_linears

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("batch,seq,heads,head", [(1, 1, 1, 8), (3, 77, 4, 64), (2, 130, 16, 128)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_rope_in_place_equals_the_eager_form(batch, seq, heads, head, dtype):
    g = torch.Generator(device=DEV).manual_seed(seq)
    c = heads * head
    table = rope_table(head, 256).to(DEV).to(dtype)
    qkv = torch.randn(batch * seq, 3 * c, device=DEV, generator=g).to(torch.bfloat16)
    q, k, v = (t.reshape(batch, seq, heads, head) for t in qkv.view(batch, seq, 3 * c).split(c, dim=2))
    q_ref, k_ref = apply_rope(q, k, table)
    v_ref = v.clone()
    assert rope_in_place_ok(qkv, table, seq, heads)
    quest.rope_inplace(qkv, table, seq, 2 * c)
    got = qkv.view(batch, seq, 3, heads, head)
    assert got[:, :, 0].equal(q_ref) and got[:, :, 1].equal(k_ref) and got[:, :, 2].equal(v_ref)
    assert not rope_in_place_ok(qkv, table, 257, heads)


@pytest.mark.parametrize("m,k", [(1, 256), (33, 2048), (130, 5632)])
@pytest.mark.parametrize("block", [64, 128, 256])
def test_producers_and_residual(m, k, block):
    g = torch.Generator(device=DEV).manual_seed(m + k)
    x, y = (torch.randn(m, k, device=DEV, generator=g).to(torch.bfloat16) for _ in range(2))
    w = (1 + 0.1 * torch.randn(k, device=DEV, generator=g)).to(torch.bfloat16)

    def outputs(int8):
        return (torch.empty(m, k if int8 else k // 2, dtype=torch.uint8, device=DEV), torch.empty(m, 1, dtype=torch.bfloat16, device=DEV),
                torch.empty(m, 1, dtype=torch.int32, device=DEV))

    def same(got, ref):
        codes, scale, sums = got
        if codes.size(1) == k:
            codes = (codes.view(torch.int8) // 16).view(m, k // 32, 2, 16).transpose(2, 3).reshape(m, k)
        else:
            codes = quest.unpack_int4(codes)
        return codes.equal(quest.unpack_int4(ref[0])) and scale.equal(ref[1]) and sums.equal(ref[2])

    norm = quest.rmsnorm_hadamard_quantize_int4(x, w, 1e-5, block)
    added = quest.rmsnorm_hadamard_quantize_int4(x + y, w, 1e-5, block)
    gate = quest.silu_mul_hadamard_quantize_int4(x, y, block)
    for int8 in (False, True):
        if int8 and k % 128:
            continue
        assert same(quest.producer_hadamard_quantize(quest.PRODUCE_RMSNORM, x, *outputs(int8), norm_weight=w, eps=1e-5, block=block), norm)
        assert same(quest.producer_hadamard_quantize(quest.PRODUCE_SILU_MUL, x, *outputs(int8), x2=y, block=block), gate)
        total, got = quest.add_rmsnorm_hadamard_quantize(x, y, w, 1e-5, *outputs(int8), block=block)
        assert total.equal(x + y) and same(got, added)


def test_fused_block_keeps_the_residual_gradient():
    torch.manual_seed(1)
    with torch.device(DEV):
        model = Decoder(DecoderConfig(n_embd=256, n_layer=2, n_head=4, ffn=512, vocab_size=64, sequence_length=32)).to(torch.bfloat16)
    swap_linears(model, "int4_fused")
    x = torch.randn(2, 17, 256, device=DEV).to(torch.bfloat16)
    with torch.no_grad():
        ref = [blk(x, model.rope) for blk in model.transformer.h]
    x.requires_grad_()
    g = torch.randn_like(x)
    for blk, y_ref in zip(model.transformer.h, ref):
        y = blk(x, model.rope)
        assert y.equal(y_ref)
        assert torch.autograd.grad(y, x, g)[0].equal(g)
    model(torch.arange(34, device=DEV).view(2, 17)).float().sum().backward()
    assert model.transformer.wte.weight.grad.abs().sum() > 0 and model.transformer.ln_f.weight.grad is not None


@pytest.mark.parametrize("m,k", [(1, 8), (37, 2048), (9, 2056), (5, 5632)])
def test_rmsnorm_kernel(m, k):
    g = torch.Generator(device=DEV).manual_seed(k)
    x = torch.randn(m, k, device=DEV, generator=g).to(torch.bfloat16)
    w = (1 + 0.1 * torch.randn(k, device=DEV, generator=g)).to(torch.bfloat16)
    y = quest.rmsnorm(x, w, 1e-5)
    xd = x.double()
    exact = xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-5) * w.double()
    # two roundings to bf16: the significand has 8 bits, half an ulp is at most 2^-8 of the value
    assert (y.double() - exact).abs().le(2 * 2.0 ** -8 * exact.abs() * 1.01 + 1e-30).all()


@pytest.mark.parametrize("c", [1.0078125, 1.4140625, 1.8046875])
@pytest.mark.parametrize("k", [2048, 65536])
def test_rmsnorm_sums_long_rows(c, k):
    """A constant row whose squares one long fp32 chain rounds down: at 2048 terms per lane (K = 65536) such a sum is 1.5e-5 to
    3e-5 low and c * rinv half of that high.  eps puts the exact quotient 0.35e-5 below the tie between the two largest bf16
    values up to 1, a margin of fifty fp32 roundings."""
    tie = 1 - 2.0 ** -9
    t = tie * (1 - 0.35e-5)
    y = quest.rmsnorm(torch.full((3, k), c, dtype=torch.bfloat16, device=DEV), torch.ones(k, dtype=torch.bfloat16, device=DEV), c * c * (t ** -2 - 1))
    assert (y == 1 - 2.0 ** -8).all()


def test_silu_quotient_keeps_every_rounding():
    """The gate of the fused quantiser against torch's silu over all bf16 values.  Every value v sits alone in a row, next to a
    factor that brings silu(v) near 1 (a power of two, exact), so that the row's scale is a rounded multiple of it; several
    multiples of the factor, because one alone maps neighbouring values to one scale here and there."""
    v = torch.arange(65536, device=DEV, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    v = v[v.isfinite()]
    s = torch.nn.functional.silu(v)
    near_one = torch.exp2((1 - torch.frexp(s.double())[1].double()).clamp(-126, 126))  # v below -88 gives -0: any factor

    def row(first, rest=0.0):
        t = torch.full((v.numel(), 64), rest, dtype=torch.bfloat16, device=DEV)
        t[:, 0] = first
        return t

    seen = {-1: torch.zeros_like(v, dtype=torch.bool), 1: torch.zeros_like(v, dtype=torch.bool)}
    for multiple in (1.0, 1.1875, 1.375, 1.5, 1.6875, 1.875):
        up = row((near_one * multiple).to(torch.bfloat16), 1.0)
        ref = quest.hadamard_quantize_int4(row(s) * up, 64)
        got = quest.silu_mul_hadamard_quantize_int4(row(v), up, 64)
        assert all(a.equal(b) for a, b in zip(got, ref)), multiple  # codes (the sign), scales, row sums
        for step in seen:  # the same row with the value one unit in the last place off
            other = (s.view(torch.int16) + step).view(torch.bfloat16)
            seen[step] |= (quest.hadamard_quantize_int4(row(other) * up, 64)[1] != ref[1]).flatten()
    nonzero = s != 0
    assert seen[-1][nonzero].all() and seen[1][nonzero].all()  # ... shows, so the comparison above can fail
