"""The int8-operand GEMM (CTA-pair kernel, few-token kernel) and the layers that take it, at the edges of their tiles."""
from __future__ import annotations

import pytest
import torch

import quest_b200 as quest

pytestmark = pytest.mark.gpu
DEV = "cuda"


def problem(m, k, n, seed, extreme=False):
    g = torch.Generator(device=DEV).manual_seed(seed)
    a = torch.randint(-8, 8, (m, k), dtype=torch.int8, device=DEV, generator=g)
    if extreme:
        a.fill_(-8)
    w = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device=DEV, generator=g)
    if extreme:
        w.fill_(0x88)
    halves = a.view(m, k // 32, 16, 2)  # the operand: sixteen times the codes, even positions of every 32 first
    a8 = (torch.cat([halves[..., 0], halves[..., 1]], dim=-1).reshape(m, k) * 16).view(torch.uint8).contiguous()
    a_add = torch.randint(-8 * k, 8 * k, (m, 1), dtype=torch.int32, device=DEV, generator=g)
    b_add = torch.randint(-8 * k, 8 * k, (n, 1), dtype=torch.int32, device=DEV, generator=g)
    a_mul = (0.01 + torch.rand(m, 1, device=DEV, generator=g)).to(torch.bfloat16)
    b_mul = (0.01 + torch.rand(n, 1, device=DEV, generator=g)).to(torch.bfloat16)
    acc = (a.double() @ quest.unpack_int4(w).double().t()).to(torch.int32)  # exact
    want = ((2 * acc + a_add + b_add.t()).float() * (0.5 * a_mul.float() * b_mul.float().t())).to(torch.bfloat16)
    return (a8, w, a_add, b_add, a_mul, b_mul), want


def check(args, want):
    out = torch.full_like(want, float("nan"))
    quest.fused_matmul_dequantize_a8(*args, out=out)
    assert quest.device_status() == 0
    assert out.equal(want)


# one row to one beyond a tile; N below a 32-column piece, ragged, odd (per-thread stores), narrow balanced columns, several
# tiles per pair with the accumulator buffers taking turns; K of one and a few steps; more than 32 tile rows (grouped walk)
@pytest.mark.parametrize("m,k,n", [(1, 128, 8), (129, 640, 24), (255, 256, 250), (256, 128, 256), (257, 1408, 5001), (1000, 384, 1032),
                                   (2048, 256, 4096), (4097, 128, 2560), (8500, 128, 1000)])
def test_pair_kernel(monkeypatch, m, k, n):
    monkeypatch.setenv("QB200_A8_KERNEL", "pair")
    args, want = problem(m, k, n, m + k + n)
    check(args, want)
    for group in ("3", "16"):
        monkeypatch.setenv("QB200_GEMM_GROUP", group)
        check(args, want)
    monkeypatch.setenv("QB200_GEMM_BALANCE", "0")
    monkeypatch.setenv("QB200_GEMM_TMA_STORE", "0")
    check(args, want)


# long reductions over many columns: over a hundred steps of the packed ring, the weights from HBM (their copies land out of
# order when memory is cold: nine sets of weights larger than L2 together take turns)
@pytest.mark.parametrize("m,k,n", [(33, 28672, 776), (130, 28672, 2048), (300, 16384, 4096), (256, 28672, 8192)])
def test_pair_kernel_long_reductions(monkeypatch, m, k, n):
    monkeypatch.setenv("QB200_A8_KERNEL", "pair")
    (a8, w, a_add, b_add, a_mul, b_mul), want = problem(m, k, n, m + k + n)
    turns = [(torch.roll(w, i, 0), torch.roll(b_add, i, 0), torch.roll(b_mul, i, 0)) for i in range(9)]
    flush = torch.empty(1 << 28, dtype=torch.uint8, device=DEV)
    for _ in range(3):
        flush.zero_()
        for i, (wi, add, mul) in enumerate(turns):
            check((a8, wi, a_add, add, a_mul, mul), torch.roll(want, i, 1))


def test_pair_and_few_token_kernels_at_the_largest_sums(monkeypatch):
    for kernel, m in (("pair", 130), ("skinny", 16)):
        monkeypatch.setenv("QB200_A8_KERNEL", kernel)
        check(*problem(m, 131072 - 128, 64, 5, extreme=True))


# every token bucket, one row to one beyond a bucket; weight rows per CTA from 8 to 128 and 1 to 8 K ranges, uneven ones too
@pytest.mark.parametrize("m", [1, 15, 16, 17, 32, 33, 64, 65, 128])
@pytest.mark.parametrize("k,n,plans", [(1152, 333, ("8,1", "120,2", "128,3", "64,8")), (5504, 1024, (None, "40,5", "128,7")),
                                       (128, 4100, (None, "128,1"))])
def test_few_token_kernel(monkeypatch, m, k, n, plans):
    monkeypatch.setenv("QB200_A8_KERNEL", "skinny")
    args, want = problem(m, k, n, m + k + n)
    for plan in plans:
        if plan is None:
            monkeypatch.delenv("QB200_SKINNY", raising=False)
        else:
            monkeypatch.setenv("QB200_SKINNY", plan)
        check(args, want)


# the layer (one call, the library's route) against the single ops on packed codes: with and without the transform, K that
# the tcgen05 quantiser cannot tile, a bias, workspaces of the caller, an output of the caller, K without an int8 route
@pytest.mark.parametrize("use_hadamard", [True, False])
@pytest.mark.parametrize("m,k,n", [(1, 4096, 512), (7, 1024, 96), (64, 5632, 264), (100, 11008, 128), (300, 2048, 1000), (1024, 4096, 256), (40, 96, 64)])
def test_layer_routes_agree(m, k, n, use_hadamard):
    if use_hadamard and k % 128:
        pytest.skip("the transform needs whole blocks")
    g = torch.Generator(device=DEV).manual_seed(m + n)
    w = (0.02 * torch.randn(n, k, device=DEV, generator=g)).to(torch.bfloat16)
    wp, ws, wa, _ = quest.preprocess_weight(w, use_hadamard=use_hadamard)
    x = torch.randn(m, k, device=DEV, generator=g).to(torch.bfloat16)
    ref = quest.linear_forward(x, wp, ws, wa, use_hadamard=use_hadamard, debug_mode=True)
    # the quantiser kernels may round a transform output the other way; the int32 sums and the epilogue may not differ
    for _ in range(2):
        y = quest.linear_forward(x, wp, ws, wa, use_hadamard=use_hadamard)
        assert (y.float() - ref.float()).norm() <= 1e-2 * ref.float().norm()
        if not use_hadamard:
            assert y.equal(ref)
    packed = torch.empty(m, k // 2, dtype=torch.uint8, device=DEV)
    scale, sums, out = torch.empty(m, 1, dtype=torch.bfloat16, device=DEV), torch.empty(m, 1, dtype=torch.int32, device=DEV), torch.empty_like(y)
    y2 = quest.linear_forward(x, wp, ws, wa, use_hadamard=use_hadamard, out=out, _a_int_packed=packed, _a_scale=scale, _a_int_row_sum=sums)
    assert y2 is out and (y2.float() - ref.float()).norm() <= 1e-2 * ref.float().norm()
    assert sums.equal(quest.unpack_int4(packed).sum(1, dtype=torch.int32, keepdim=True))
    if k % 128 == 0:
        a8 = torch.empty(m, k, dtype=torch.uint8, device=DEV)
        y3 = quest.linear_forward(x, wp, ws, wa, use_hadamard=use_hadamard, _a_int8=a8, _a_scale=scale, _a_int_row_sum=sums)
        codes = (a8.view(torch.int8) // 16).view(m, k // 32, 2, 16).transpose(2, 3).reshape(m, k)
        assert sums.equal(codes.sum(1, dtype=torch.int32, keepdim=True)) and (y3.float() - ref.float()).norm() <= 1e-2 * ref.float().norm()
    if m > 1:  # a strided activation still meets the single ops' own checks
        with pytest.raises(AssertionError):
            quest.linear_forward(torch.cat([x, x], dim=1)[:, :k], wp, ws, wa, use_hadamard=use_hadamard)
    assert quest.device_status() == 0


def test_preference_of_the_separate_ops():
    """The layer's rule, for what the tcgen05 quantiser tiles and is the faster quantiser for."""
    for m, k, n, prefers in ((1024, 2048, 6144, False), (16, 4096, 4096, False), (2048, 5632, 2048, False), (768, 4096, 4096, True),
                             (16384, 4096, 4096, True), (65536, 4096, 1024, False)):
        assert quest.prefers_a8(m, k, n) == prefers, (m, k, n)
