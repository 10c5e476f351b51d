"""Layer logic on top of the ops: weight preparation, the W4A4 linear forward and the module.

Mirrors the dense branches of gemm-quest/benchmarks/utils.py (``preprocess_weight`` :20-53,
``linear_forward`` :56-111, ``unpack_int4`` :420-445) and ``Linear4bit`` of
gemm-quest/benchmarks/bench_e2e.py:41-70, without the backend switch (there is one backend) and without
the 4:8-sparse branch.  With ``use_hadamard`` the activation side is ONE fused kernel
(Hadamard + scale + quantise + pack + row sum) followed by the fused GEMM: two launches per layer
instead of the reference's four.
"""
from __future__ import annotations

import torch
from torch import nn
from torch.autograd import forward_ad

import quest_b200 as quest
from . import _lib
from .workspace import default_cache, layer_workspaces

HADAMARD_BLOCK = 128  # the reference hard-codes block 128 (utils.py:17, 39, 90)


def preprocess_weight(
        weight: torch.Tensor,
        use_sparse: bool = False,
        use_hadamard: bool = False,
        backend: str = 'cuda',
        block: int = HADAMARD_BLOCK,
) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor | None]:
    """weight bf16 (N, K) -> (w_int_packed u8 (N, K//2), w_scale bf16 (N, 1), w_add i32 (N, 1), None).

    ``w_add = row_sum + K // 2`` folds the +0.5 offsets of both operands into the epilogue
    (utils.py:48).  ``backend`` is accepted for signature compatibility and ignored.
    """
    if use_sparse:
        raise NotImplementedError("quest_b200 implements the dense W4A4 path only")
    weight = weight.contiguous()
    if quest.one_pass_ok(weight, block if use_hadamard else 0):
        w_int_packed, w_scale, w_add = quest.scale_quantize_int4(weight, weight_block=block if use_hadamard else 0,
                                                                 row_sum_add=weight.size(1) // 2)
        return w_int_packed, w_scale, w_add, None
    if use_hadamard:
        weight = quest.hadamard_transform(weight, block=block, weight_side=True)
    N, K = weight.shape
    w_scale = torch.empty(N, 1, dtype=weight.dtype, device=weight.device)
    w_int_packed = torch.empty(N, K // 2, dtype=torch.uint8, device=weight.device)
    w_int_row_sum = torch.empty(N, 1, dtype=torch.int32, device=weight.device)
    quest.find_scale_int4(x=weight, scale=w_scale)
    quest.quantize_int4(x=weight, scale=w_scale, x_int=None, x_int_packed=w_int_packed,
                        x_int_row_sum=w_int_row_sum, do_dequantize=False)
    w_add = w_int_row_sum + K // 2
    return w_int_packed, w_scale, w_add, None


def fused_matmul_dequantize_int4_bf16(
        mat_a: torch.Tensor,
        mat_b: torch.Tensor,
        vec_a_add: torch.Tensor,
        vec_b_add: torch.Tensor,
        vec_a_mul: torch.Tensor,
        vec_b_mul: torch.Tensor,
        mat_d: torch.Tensor,
        _mat_c: torch.Tensor = None,
        debug_mode: bool = True,
) -> torch.Tensor:
    """mat_d (M, N) bf16 = (2 * mat_a @ mat_b^T + vec_a_add + vec_b_add^T) * (.5 * vec_a_mul * vec_b_mul^T).

    The switch of gemm-quest/benchmarks/utils.py:548-587: ``debug_mode=True`` (the reference's default) takes the
    unfused route - int32 GEMM into ``_mat_c`` (allocated if absent), then ``add_mul_vv`` - and ``debug_mode=False``
    the fused kernel.  Here both routes evaluate the same exact expression, so their results are bit-identical.
    ``mat_d`` may be None (allocated in the dtype of ``vec_a_mul``)."""
    M, N = mat_a.size(0), mat_b.size(0)
    device = mat_a.device
    if mat_d is None:
        mat_d = torch.empty(M, N, dtype=vec_a_mul.dtype, device=device)
    if debug_mode:
        mat_c = torch.empty(M, N, dtype=torch.int32, device=device) if _mat_c is None else _mat_c
        quest.matmul_int4_int4t_int32(mat_a=mat_a, mat_b=mat_b, out=mat_c)
        quest.add_mul_vv(vec_a_add=vec_a_add, vec_a_mul=vec_a_mul, vec_b_add=vec_b_add, vec_b_mul=vec_b_mul,
                         mat_c=mat_c, mat_d=mat_d)
    else:
        quest.fused_matmul_dequantize_int4_int4t_bf16(mat_a=mat_a, mat_b=mat_b, vec_a_add=vec_a_add, vec_b_add=vec_b_add,
                                                      vec_a_mul=vec_a_mul, vec_b_mul=vec_b_mul, out=mat_d)
    return mat_d


_BLOCKS = (64, 128, 256)


def _caller_workspaces(x, n, a_int8, a_int_packed, a_scale, a_sums):
    """(codes, scale, row sums) for ``_layer_call`` from what the caller gave, the missing ones allocated; None if nothing was
    given.  Of two code buffers the one the library's own choice needs is used."""
    if a_int8 is None and a_int_packed is None and a_scale is None and a_sums is None:
        return None
    m, k = x.shape
    codes = a_int_packed if a_int8 is None else a_int8
    if (a_int8 is None) == (a_int_packed is None):
        int8 = quest.layer_operand(m, k, n)
        codes = torch.empty(m, k if int8 else k // 2, dtype=torch.uint8, device=x.device) if codes is None else a_int8 if int8 else a_int_packed
    return (codes, torch.empty(m, 1, dtype=x.dtype, device=x.device) if a_scale is None else a_scale,
            torch.empty(m, 1, dtype=torch.int32, device=x.device) if a_sums is None else a_sums)


def _layer_call(x, w, w_scale, w_add, out, ws, block, bias=None):
    """The whole layer as one library call, or None where its buffers are not what that call takes (linear_forward then goes
    through the single ops, which check and report).  ``block`` 0: no transform.  ``ws``: None, or (codes, scale, row sums)
    where codes [M, K] selects the int8 operand and [M, K/2] packed int4; None takes one allocation for all three.
    ``bias``: added as ``y += bias`` would, in the GEMM's epilogue where it can."""
    if x.dim() != 2 or w.dim() != 2 or not x.is_cuda:
        return None
    (m, k), n, dev = x.shape, w.size(0), x.get_device()
    if (m == 0 or n == 0 or k == 0 or k > 65536 or w.size(1) * 2 != k or (k % block if block else k % 32)
            or x.dtype is not torch.bfloat16 or w.dtype is not torch.uint8 or w_scale.dtype is not torch.bfloat16
            or w_add.dtype is not torch.int32 or w_scale.numel() < n or w_add.numel() < n
            or w.get_device() != dev or w_scale.get_device() != dev or w_add.get_device() != dev
            or not (x.is_contiguous() and w.is_contiguous() and w_scale.is_contiguous() and w_add.is_contiguous())):
        return None
    xp, wp = x.data_ptr(), w.data_ptr()
    if xp % 16 or wp % 16:
        return None
    if out is None:
        out = x.new_empty((m, n))
    elif out.shape != (m, n) or out.dtype is not torch.bfloat16 or out.get_device() != dev or not out.is_contiguous():
        return None
    lib = _lib.load()
    if ws is None:
        int8 = lib.quest_b200_layer_plan(m, k, n, block)
        if int8 == 2:  # one kernel, no workspace
            codes = sums = scale = None
        else:
            code_bytes = -(-(m * k if int8 else m * (k // 2)) // 256) * 256
            try:
                buf = x.new_empty(code_bytes // 2 + 3 * m)  # bf16 elements: two bytes each
            except torch.OutOfMemoryError:  # a layer fits where its packed form does
                if not int8:
                    raise
                int8, code_bytes = 0, -(-(m * (k // 2)) // 256) * 256
                buf = x.new_empty(code_bytes // 2 + 3 * m)
            codes = buf.data_ptr()
            sums = codes + code_bytes
            scale = sums + 4 * m
    else:
        a, a_scale, a_sums = ws
        if (a.shape not in ((m, k), (m, k // 2)) or a.dtype is not torch.uint8 or a_scale.dtype is not torch.bfloat16
                or a_sums.dtype is not torch.int32 or a_scale.numel() < m or a_sums.numel() < m
                or a.get_device() != dev or a_scale.get_device() != dev or a_sums.get_device() != dev
                or not (a.is_contiguous() and a_scale.is_contiguous() and a_sums.is_contiguous()) or a.data_ptr() % 16):
            return None
        int8 = int(a.size(1) == k)
        codes, scale, sums = a.data_ptr(), a_scale.data_ptr(), a_sums.data_ptr()
    if int8 == 1 and k % 128:
        return None
    late_bias = None  # a bias that autograd follows is added by torch
    if bias is not None and not (not (bias.requires_grad and torch.is_grad_enabled()) and forward_ad._current_level < 0 and bias.dtype is torch.bfloat16 and bias.dim() == 1 and bias.size(0) == n and bias.get_device() == dev
                                 and bias.is_contiguous() and lib.quest_b200_layer_adds_bias(m, k, n, int8)):
        bias, late_bias = None, bias
    args = (out.data_ptr(), xp, wp, w_add.data_ptr(), w_scale.data_ptr(), None if bias is None else bias.data_ptr(), codes, int8, scale, sums, m, k, n, block,
            torch._C._cuda_getCurrentRawStream(dev))
    if torch._C._cuda_getDevice() == dev:
        status = lib.w4a4_linear_layer_cuda(*args)
    else:
        with torch.cuda.device(dev):
            status = lib.w4a4_linear_layer_cuda(*args)
    if status:
        _lib.check(status, "w4a4_linear_layer_cuda")
    if late_bias is not None:
        out += late_bias
    return out


def linear_forward(
        activation: torch.Tensor,
        w_int_packed: torch.Tensor,
        w_scale: torch.Tensor,
        w_add: torch.Tensor,
        w_meta_e: torch.Tensor = None,
        out: torch.Tensor = None,
        _a_scale: torch.Tensor = None,
        _a_int_packed: torch.Tensor = None,
        _a_int_row_sum: torch.Tensor = None,
        _c: torch.Tensor = None,
        use_hadamard: bool = False,
        backend: str = 'cuda',
        block: int = HADAMARD_BLOCK,
        _a_int8: torch.Tensor = None,
        debug_mode: bool = False,
) -> torch.Tensor:
    """out (M, N) bf16 = activation (M, K) @ weight^T in W4A4.  The ``_a_*`` arguments are optional
    caller-owned workspaces (CUDA-graph friendly), as in the reference.  As in the reference (utils.py:100) the
    fused kernel is used whether or not ``_c`` is given; ``debug_mode=True`` (not in the reference's signature)
    takes the unfused int32 GEMM + add_mul_vv route with ``_c`` as its int32 workspace.

    Where the library finds it faster the quantiser writes the GEMM's int8 operand directly (``_a_int8`` [M, K] uint8 is its
    workspace) instead of packed int4: same codes, same result, no unpack of A inside the GEMM.  A caller that passes
    ``_a_int_packed`` but no ``_a_int8`` keeps the packed route; of both, the one of the library's choice is written.

    With dense buffers the layer is ONE library call (``_layer_call``): the quantiser (with or without the transform, each
    row read once), then the GEMM kernel, where it pays launched with a programmatic dependency on the quantiser so that
    its set-up and first weight copies overlap the quantiser's end."""
    if w_meta_e is not None:
        raise NotImplementedError("quest_b200 implements the dense W4A4 path only")
    if not debug_mode and activation.dim() == 2 and (not use_hadamard or block in _BLOCKS):
        ws = _caller_workspaces(activation, w_int_packed.size(0), _a_int8, _a_int_packed, _a_scale, _a_int_row_sum)
        y = _layer_call(activation, w_int_packed, w_scale, w_add, out, ws, block if use_hadamard else 0)
        if y is not None:
            return y
    M, K, N = activation.size(0), activation.size(1), w_int_packed.size(0)
    dtype, device = activation.dtype, activation.device
    if out is None:
        out = torch.empty(M, N, dtype=dtype, device=device)
    a_scale = torch.empty(M, 1, dtype=dtype, device=device) if _a_scale is None else _a_scale
    a_int_row_sum = torch.empty(M, 1, dtype=torch.int32, device=device) if _a_int_row_sum is None else _a_int_row_sum
    a_int_packed = torch.empty(M, K // 2, dtype=torch.uint8, device=device) if _a_int_packed is None else _a_int_packed
    assert w_int_packed.size(1) * 2 == K and (debug_mode or not use_hadamard or out.shape == (M, N))
    if use_hadamard:
        quest.hadamard_quantize_int4(activation, block=block, x_int_packed=a_int_packed, scale=a_scale,
                                     x_int_row_sum=a_int_row_sum)
    else:
        quest.find_scale_int4(x=activation, scale=a_scale)
        quest.quantize_int4(x=activation, scale=a_scale, x_int=None, x_int_packed=a_int_packed,
                            x_int_row_sum=a_int_row_sum, do_dequantize=False)
    fused_matmul_dequantize_int4_bf16(mat_a=a_int_packed, mat_b=w_int_packed, vec_a_add=a_int_row_sum, vec_b_add=w_add,
                                      vec_a_mul=a_scale, vec_b_mul=w_scale, mat_d=out, _mat_c=_c, debug_mode=debug_mode)
    return out


def unpack_int4(x_int_packed: torch.Tensor) -> torch.Tensor:
    """uint8 (..., K // 2) -> int8 codes (..., K); test helper, plain torch (utils.py:420-445)."""
    x_int = torch.empty(*x_int_packed.shape[:-1], x_int_packed.size(-1) * 2, dtype=torch.int8,
                        device=x_int_packed.device)
    x_int[..., ::2] = x_int_packed & 0xF
    x_int[..., 1::2] = x_int_packed >> 4
    return torch.where(x_int >= 8, x_int - 16, x_int)


class Linear4bit(nn.Module):
    """nn.Linear whose weight is stored as packed int4 + per-row scale/offset and whose forward runs
    the W4A4 kernels (gemm-quest/benchmarks/bench_e2e.py:41-70).  Needs a CUDA device."""

    def __init__(self, in_features: int, out_features: int, bias: bool = True, device=None, dtype=None,
                 use_sparse: bool = False, use_hadamard: bool = False, use_noop: bool = False,
                 weight: torch.Tensor | None = None):
        super().__init__()
        self.in_features, self.out_features = in_features, out_features
        self.use_hadamard: bool = use_hadamard
        self.use_noop: bool = use_noop
        self.workspaces = default_cache  # a WorkspaceCache; replace it to give a module (or a model) its own
        nn_linear = nn.Linear(in_features, out_features, bias=bias, device=device, dtype=dtype)
        if weight is not None:
            nn_linear.weight.data.copy_(weight)
        self.bias = nn_linear.bias
        w = nn_linear.weight.data
        self.weight = torch.empty_like(w, device=torch.device('meta'))
        w_int_packed, w_scale, w_add, w_meta_e = preprocess_weight(weight=w, use_sparse=use_sparse,
                                                                   use_hadamard=use_hadamard)
        self.register_buffer('w_int_packed', w_int_packed)
        self.register_buffer('w_scale', w_scale)
        self.register_buffer('w_add', w_add)
        self.register_buffer('w_meta_e', w_meta_e)

    def forward_quantized(self, a_int_packed: torch.Tensor, a_scale: torch.Tensor, a_int_row_sum: torch.Tensor,
                          out: torch.Tensor = None) -> torch.Tensor:
        """The layer on activations that are already quantised ([M, K/2] packed codes, [M, 1] scales and row sums, as
        written by ``hadamard_quantize_int4`` or one of its producer-fused variants): only the fused GEMM runs.  Several
        layers that read the same activations (w1 and w2 of a SwiGLU block) can share one quantisation this way.
        ``a_int_packed`` [M, K] instead of [M, K/2] is the int8 operand (``producer_hadamard_quantize``)."""
        if a_int_packed.size(1) == self.in_features:
            y = quest.fused_matmul_dequantize_a8(mat_a8=a_int_packed, mat_b=self.w_int_packed, vec_a_add=a_int_row_sum,
                                                 vec_b_add=self.w_add, vec_a_mul=a_scale, vec_b_mul=self.w_scale, out=out)
            if self.bias is not None:
                y += self.bias
            return y
        y = quest.fused_matmul_dequantize_int4_int4t_bf16(mat_a=a_int_packed, mat_b=self.w_int_packed, vec_a_add=a_int_row_sum,
                                                          vec_b_add=self.w_add, vec_a_mul=a_scale, vec_b_mul=self.w_scale, out=out)
        if self.bias is not None:
            y += self.bias
        return y

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        if not self.use_noop:
            a = x.contiguous()
            if a.dim() != 2:
                a = a.flatten(end_dim=-2)
            # activation-side workspaces come from the shared per-stream cache: nothing but the output is allocated
            m, k = a.shape
            block = HADAMARD_BLOCK if self.use_hadamard else 0
            plan = _lib.load().quest_b200_layer_plan(m, k, self.out_features, block)
            out = a.new_empty((m, self.out_features))  # before the workspaces, which have a smaller form where memory is short
            ws, buffers = {}, None
            if plan != 2:
                ws = layer_workspaces(self.workspaces, m, k, a.device, a.dtype, plan == 1)
                buffers = (ws["_a_int8"] if "_a_int8" in ws else ws["_a_int_packed"], ws["_a_scale"], ws["_a_int_row_sum"])
            y = _layer_call(a, self.w_int_packed, self.w_scale, self.w_add, out, buffers, block, self.bias)
            if y is not None:
                return y if x.dim() == 2 else y.view(*x.shape[:-1], self.out_features)
            y = linear_forward(activation=a, w_int_packed=self.w_int_packed, w_scale=self.w_scale, w_add=self.w_add,
                               w_meta_e=self.w_meta_e, out=None, use_hadamard=self.use_hadamard, **ws)
            y = y.unflatten(dim=0, sizes=x.shape[:-1])
        else:
            if self.use_hadamard:
                x = quest.hadamard_transform(x.contiguous(), block=HADAMARD_BLOCK, weight_side=True)
            y = torch.zeros(*x.shape[:-1], self.out_features, dtype=x.dtype, device=x.device)
        if self.bias is not None:
            y += self.bias
        return y
