"""Functional front-end of the hot operators (autograd wrappers).

Each function dispatches to the native sm_100a kernels for CUDA tensors and to the PyTorch
reference otherwise (see :mod:`libai_b200.ops`).  The reference call sites these replace are the
OneFlow fused ops ``flow._C.layer_norm_affine`` / ``rms_norm``
(libai/layers/layer_norm.py:78-131), ``fused_bias_add_gelu`` (libai/layers/mlp.py:95),
``fused_bias_add_dropout`` (libai/layers/mlp.py:104, attention.py:265),
``fused_scale_mask_softmax_dropout`` / ``fused_scale_tril_softmax_mask_scale``
(libai/layers/attention.py:220-246), ``sparse_softmax_cross_entropy``
(libai/layers/cross_entropy.py:44) and the matmuls in libai/layers/linear.py:123-157.
"""
from __future__ import annotations

import math
from typing import Optional, Tuple

import torch
import torch.distributed as dist
import torch.nn.functional as F
from torch._subclasses.fake_tensor import FakeTensor

from . import count_launch, load_ext, use_native
from .. import ops


def _plain_call() -> bool:
    """False where an operator is transformed (vmap, jvp, …), differentiated forward or traced: those see PyTorch operators.  Asked (like the
    type of a tensor without memory, ``FakeTensor``) before anything looks at an address."""
    return not (torch._C._are_functorch_transforms_active() or torch.autograd.forward_ad._current_level >= 0 or torch.jit.is_tracing())


class _NoGradContext:
    """Stands in for the context of an autograd function whose backward will never run: keeps nothing."""

    needs_input_grad = (False,) * 32

    def save_for_backward(self, *tensors):
        pass


def _call(fn, *args):
    """``fn.apply(*args)``; where no graph is recorded the forward alone (an ``apply`` costs ~10 us of host time, more than most
    kernels of a generation step take)."""
    if torch.is_grad_enabled() or not _plain_call():
        return fn.apply(*args)
    return fn.forward(_NoGradContext(), *args)


_PLAIN_TYPES = (torch.Tensor, torch.nn.Parameter)


def _graph_node(*tensors) -> bool:
    """Does this call record a graph that the C++ nodes (csrc/autograd_nodes.cpp) can stand for?  Not where a call is transformed, traced or compiled or a
    dispatch mode looks at its operators, not for subclasses, not for fp8 products: those take the autograd functions below."""
    if not torch.is_grad_enabled() or ops.fp8_enabled() or not _plain_call() or torch._C._len_torch_dispatch_stack() or torch.compiler.is_compiling():
        return False
    for t in tensors:
        if t is not None and (type(t) not in _PLAIN_TYPES or not t.is_cuda):
            return False
    return True


# --------------------------------------------------------------------------------------
# activations (reference math)
# --------------------------------------------------------------------------------------
_SQRT_2_OVER_PI = 0.7978845608028654


def gelu_ref(x, approximate: str = "none"):
    return F.gelu(x, approximate=approximate)


ACT_NONE, ACT_GELU, ACT_GELU_TANH, ACT_RELU, ACT_SILU, ACT_QUICK_GELU = 0, 1, 2, 3, 4, 5
_ACT_IDS = {
    None: ACT_NONE,
    "none": ACT_NONE,
    "gelu": ACT_GELU,
    "gelu_tanh": ACT_GELU_TANH,
    "relu": ACT_RELU,
    "silu": ACT_SILU,
    "quick_gelu": ACT_QUICK_GELU,
}


def _act_ref(x, act):
    if act in (None, "none"):
        return x
    if act == "gelu":
        return F.gelu(x)
    if act == "gelu_tanh":
        return F.gelu(x, approximate="tanh")
    if act == "relu":
        return F.relu(x)
    if act == "silu":
        return F.silu(x)
    if act == "quick_gelu":
        return x * torch.sigmoid(1.702 * x)
    raise ValueError(act)


# --------------------------------------------------------------------------------------
# GEMM: y = x @ w^T (+ bias) (+ activation)
# --------------------------------------------------------------------------------------
def _gemm_ok(x: torch.Tensor, w: torch.Tensor) -> bool:
    """Shapes/dtypes the tcgen05 kernel accepts (TMA needs 16-byte aligned rows)."""
    return (
        x.dtype == torch.bfloat16
        and w.dtype == torch.bfloat16
        and x.shape[-1] % 8 == 0
        and w.shape[0] % 8 == 0
        and x.numel() > 0
    )



_FP8_WEIGHTS: dict = {}


def _fp8_ok(x2: torch.Tensor, w: torch.Tensor) -> bool:
    return ops.fp8_enabled() and x2.shape[-1] % 16 == 0 and w.is_contiguous()


def _fp8_weight(ext, w):
    """E4M3 copy of a weight + its dequantisation scale, cached until the optimizer rewrites the parameters
    (``ops.bump_fp8_weight_epoch``) or the tensor is modified through PyTorch (``_version``).  Inside a CUDA-graph
    capture the quantisation is always issued (and captured): a cached tensor would pin stale addresses."""
    if torch.cuda.is_current_stream_capturing():
        count_launch(2)
        return ext.quantize_e4m3(w.detach())
    key = (ops.fp8_weight_epoch(), w._version, w.data_ptr())
    hit = _FP8_WEIGHTS.get(id(w))
    if hit is not None and hit[0] == key:
        return hit[1], hit[2]
    wq, dw = ext.quantize_e4m3(w.detach())
    count_launch(2)
    _FP8_WEIGHTS[id(w)] = (key, wq, dw)
    return wq, dw


def _linear_fwd_any(ext, x2, w, bias, act_id, need_pre, residual=None):
    """Forward GEMM of a linear layer: E4M3 operands when the fp8 path is on, bf16 otherwise."""
    if _fp8_ok(x2, w):
        xq, dx = ext.quantize_e4m3(x2)
        wq, dw = _fp8_weight(ext, w)
        count_launch(3)
        return ext.linear_fp8_fwd(xq, wq, dx, dw, bias, act_id, need_pre, residual)
    count_launch()
    if residual is not None:
        return ext.linear_bias_residual(x2, w, bias, residual), None
    return ext.linear_fwd(x2, w, bias, act_id, need_pre)


def _bias_grad(ext, g2, bias):
    """Column sums of ``g2`` as the gradient of ``bias``: accumulated straight into ``bias.main_grad`` (fp32 slice of
    the optimizer's flat gradient buffer) when the parameter owns one – no temporary, no bf16 round trip, no
    per-parameter add kernel later – otherwise returned as a tensor for autograd."""
    count_launch()
    main_grad = getattr(bias, "main_grad", None)
    if main_grad is not None and main_grad.dtype == torch.float32:
        ext.colsum(g2, main_grad)
        bias.grad_added_to_main_grad = True
        return None
    return ext.colsum(g2).to(bias.dtype)


class _LinearFn(torch.autograd.Function):
    """Native linear: fwd ``NT`` GEMM with fused bias/activation epilogue, dgrad ``NN`` GEMM,
    wgrad ``TN`` split-K GEMM accumulating in fp32 straight into ``weight.main_grad`` when the
    parameter owns one (gradient-accumulation fusion)."""

    @staticmethod
    def forward(ctx, x, w, bias, act):
        ext = load_ext()
        x2 = x.reshape(-1, x.shape[-1])
        if not x2.is_contiguous():
            x2 = x2.contiguous()
        need_pre = act not in (None, "none") and any(ctx.needs_input_grad[:2])
        y, pre = _linear_fwd_any(ext, x2, w, bias, _ACT_IDS[act], need_pre)
        ctx.act = act
        ctx.has_bias = bias is not None
        ctx.bias_param = bias
        ctx.save_for_backward(x2, w, pre if need_pre else None)
        ctx.x_shape = x.shape
        return y.view(*x.shape[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, gy):
        ext = load_ext()
        x2, w, pre = ctx.saved_tensors
        g2 = gy.reshape(-1, gy.shape[-1])
        if not g2.is_contiguous():
            g2 = g2.contiguous()
        if ctx.act not in (None, "none"):
            g2 = ext.act_bwd(g2, pre, _ACT_IDS[ctx.act])
            count_launch()
        gx = gw = gb = None
        if ctx.needs_input_grad[0]:
            gx = ext.gemm(g2, w, 1, None, None, False, torch.bfloat16)  # NN: [M,N]x[N,K]
            count_launch()
            gx = gx.view(ctx.x_shape)
        if ctx.needs_input_grad[1]:
            main_grad = getattr(w, "main_grad", None)
            if main_grad is not None:
                ext.gemm(g2, x2, 2, None, main_grad, True, torch.float32)  # TN accumulate
                gw = None
                w.grad_added_to_main_grad = True
            else:
                gw = ext.gemm(g2, x2, 2, None, None, False, torch.float32).to(w.dtype)
            count_launch()
        if ctx.has_bias and ctx.needs_input_grad[2]:
            gb = _bias_grad(ext, g2, ctx.bias_param)
        return gx, gw, gb, None


def linear(x, w, bias=None, act: Optional[str] = None):
    """``act(x @ w.T + bias)``; ``w`` is ``[out, in]``."""
    if use_native(x, w) and _gemm_ok(x, w):
        if _graph_node(x, w, bias):
            return load_ext().linear_node(x, w, bias, _ACT_IDS[act])
        return _call(_LinearFn, x, w, bias, act)
    y = F.linear(x, w.to(x.dtype) if w.dtype != x.dtype else w, None if bias is None else bias.to(x.dtype))
    return _act_ref(y, act)



class _MLPFn(torch.autograd.Function):
    """``act(x @ w1ᵀ + b1) @ w2ᵀ`` as one autograd node so the backward can fuse across the two GEMMs:
    ``dpre = (dy @ w2) ⊙ act'(pre)`` is a single kernel (activation backward in the dgrad epilogue) – the
    separate bias+activation backward pass over the ``[tokens, ffn]`` tensor disappears."""

    @staticmethod
    def forward(ctx, x, w1, b1, w2, act, b2=None, residual=None):
        ext = load_ext()
        x2 = x.reshape(-1, x.shape[-1])
        if not x2.is_contiguous():
            x2 = x2.contiguous()
        h, pre = _linear_fwd_any(ext, x2, w1, b1, _ACT_IDS[act], any(ctx.needs_input_grad))
        # with a residual, the second bias and the block's residual add ride in the epilogue of the second GEMM
        res2 = residual.reshape(-1, w2.shape[0]).contiguous() if residual is not None else None
        y, _ = _linear_fwd_any(ext, h, w2, b2, 0, False, res2)
        ctx.act = act
        ctx.save_for_backward(x2, w1, w2, pre, h)
        ctx.x_shape = x.shape
        ctx.has_bias = b1 is not None
        ctx.bias_param = b1
        ctx.bias2_param = b2
        ctx.has_res = residual is not None
        return y.view(*x.shape[:-1], w2.shape[0])

    @staticmethod
    def backward(ctx, gy):
        ext = load_ext()
        x2, w1, w2, pre, h = ctx.saved_tensors
        g2 = gy.reshape(-1, gy.shape[-1])
        if not g2.is_contiguous():
            g2 = g2.contiguous()
        # bias gradient of the first linear = column sums of dpre: accumulated into b1.main_grad by the dgrad epilogue
        # (red.add from the staged chunk) instead of a separate pass over the [tokens, ffn] tensor
        b1 = ctx.bias_param
        fused_gb1 = None
        if ctx.has_bias and ctx.needs_input_grad[2] and ops.fused_bias_grad():
            mg = getattr(b1, "main_grad", None)
            if mg is not None and mg.dtype == torch.float32 and mg.is_contiguous():
                fused_gb1 = mg
        dpre = ext.dgrad_actgrad(g2, w2, pre, _ACT_IDS[ctx.act], fused_gb1)
        count_launch()

        def wgrad(g, inp, w):
            main_grad = getattr(w, "main_grad", None)
            count_launch()
            if main_grad is not None:
                ext.gemm(g, inp, 2, None, main_grad, True, torch.float32)
                w.grad_added_to_main_grad = True
                return None
            return ext.gemm(g, inp, 2, None, None, False, torch.float32).to(w.dtype)

        gw2 = wgrad(g2, h, w2) if ctx.needs_input_grad[3] else None
        gw1 = wgrad(dpre, x2, w1) if ctx.needs_input_grad[1] else None
        gb1 = None
        if fused_gb1 is not None:
            b1.grad_added_to_main_grad = True
        elif ctx.has_bias and ctx.needs_input_grad[2]:
            gb1 = _bias_grad(ext, dpre, ctx.bias_param)
        gx = None
        if ctx.needs_input_grad[0]:
            gx = ext.gemm(dpre, w1, 1, None, None, False, torch.bfloat16).view(ctx.x_shape)
            count_launch()
        gb2 = None
        if ctx.bias2_param is not None and ctx.needs_input_grad[5]:
            gb2 = _bias_grad(ext, g2, ctx.bias2_param)
        return gx, gw1, gb1, gw2, None, gb2, (gy if ctx.has_res else None)


def mlp(x, w1, b1, w2, act: str = "gelu", b2=None, residual=None):
    """``act(x @ w1ᵀ + b1) @ w2ᵀ``; with ``residual`` also ``+ b2 + residual`` in the second GEMM's epilogue
    (without it the second bias is left to the fused bias+dropout+residual op)."""
    if use_native(x, w1) and _gemm_ok(x, w1) and _gemm_ok(x.new_empty(1, w1.shape[0]), w2):
        if _graph_node(x, w1, b1, w2, b2, residual):
            return load_ext().mlp_node(x, w1, b1, w2, _ACT_IDS[act], None if residual is None else b2, residual, ops.fused_bias_grad())
        if residual is not None:
            return _call(_MLPFn, x, w1, b1, w2, act, b2, residual)
        return _call(_MLPFn, x, w1, b1, w2, act)
    y = linear(linear(x, w1, b1, act), w2, b2)
    return y if residual is None else y + residual


class _LinearResidualFn(torch.autograd.Function):
    """``x @ wᵀ + bias + residual`` with bias and residual added in the GEMM epilogue."""

    @staticmethod
    def forward(ctx, x, w, bias, residual):
        ext = load_ext()
        x2 = x.reshape(-1, x.shape[-1])
        if not x2.is_contiguous():
            x2 = x2.contiguous()
        y, _ = _linear_fwd_any(ext, x2, w, bias, 0, False, residual.reshape(-1, w.shape[0]).contiguous())
        ctx.bias_param = bias
        ctx.save_for_backward(x2, w)
        ctx.x_shape = x.shape
        return y.view(*x.shape[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, gy):
        ext = load_ext()
        x2, w = ctx.saved_tensors
        g2 = gy.reshape(-1, gy.shape[-1])
        if not g2.is_contiguous():
            g2 = g2.contiguous()
        gx = gw = gb = None
        if ctx.needs_input_grad[0]:
            gx = ext.gemm(g2, w, 1, None, None, False, torch.bfloat16).view(ctx.x_shape)
            count_launch()
        if ctx.needs_input_grad[1]:
            main_grad = getattr(w, "main_grad", None)
            if main_grad is not None:
                ext.gemm(g2, x2, 2, None, main_grad, True, torch.float32)
                w.grad_added_to_main_grad = True
            else:
                gw = ext.gemm(g2, x2, 2, None, None, False, torch.float32).to(w.dtype)
            count_launch()
        if ctx.bias_param is not None and ctx.needs_input_grad[2]:
            gb = _bias_grad(ext, g2, ctx.bias_param)
        return gx, gw, gb, gy


def linear_bias_residual(x, w, bias, residual):
    """``x @ wᵀ + bias + residual`` (output projection of a block, dropout-free)."""
    if use_native(x, w) and _gemm_ok(x, w) and residual is not None and residual.dtype == torch.bfloat16:
        if _graph_node(x, w, bias, residual):
            return load_ext().linear_residual_node(x, w, bias, residual)
        return _call(_LinearResidualFn, x, w, bias, residual)
    y = linear(x, w, bias)
    return y if residual is None else y + residual


def matmul_nt(a, b):
    """``a @ b.T`` without autograd bookkeeping beyond PyTorch's (used by LM head on ref path)."""
    return linear(a, b)


# --------------------------------------------------------------------------------------
# LayerNorm / RMSNorm (optionally fused with the preceding residual add)
# --------------------------------------------------------------------------------------
class _LayerNormFn(torch.autograd.Function):
    """``with_skip``: additionally return the input itself as a second output.  A pre-LN block uses the same tensor for
    the norm and for the skip connection; autograd would sum the two gradients with a separate kernel — here both
    arrive in one ``backward`` call and the skip gradient is added inside the LayerNorm backward kernel."""

    @staticmethod
    def forward(ctx, x, weight, bias, eps, rms, with_skip=False):
        ext = load_ext()
        x2 = x.reshape(-1, x.shape[-1]).contiguous()
        y, mean, rstd = ext.norm_fwd(x2, weight, bias, eps, rms)
        count_launch()
        ctx.save_for_backward(x2, weight, mean, rstd)
        ctx.rms = rms
        ctx.has_bias = bias is not None
        ctx.bias_param = bias
        ctx.with_skip = with_skip
        if with_skip:
            return y.view(x.shape), x.view_as(x)
        return y.view(x.shape)

    @staticmethod
    def backward(ctx, gy, gskip=None):
        ext = load_ext()
        x2, weight, mean, rstd = ctx.saved_tensors
        if gy is None:          # only the skip output was used
            return gskip, None, None, None, None, None
        g2 = gy.reshape(-1, gy.shape[-1]).contiguous()
        gadd = None if gskip is None else gskip.reshape(-1, gskip.shape[-1]).contiguous()
        count_launch(2)
        wg = getattr(weight, "main_grad", None)
        bg = getattr(ctx.bias_param, "main_grad", None) if ctx.has_bias else None
        if wg is not None and wg.dtype == torch.float32 and (not ctx.has_bias or bg is not None):
            # dγ / dβ are reduced straight into the fp32 main-grad slices (one kernel for both)
            gx, _, _ = ext.norm_bwd(g2, x2, weight, mean, rstd, ctx.rms, ctx.has_bias, wg, bg, gadd)
            weight.grad_added_to_main_grad = True
            if ctx.has_bias:
                ctx.bias_param.grad_added_to_main_grad = True
            return gx.view(gy.shape), None, None, None, None, None
        gx, gw, gb = ext.norm_bwd(g2, x2, weight, mean, rstd, ctx.rms, ctx.has_bias, None, None, gadd)
        return (gx.view(gy.shape), gw.to(weight.dtype), (gb.to(weight.dtype) if ctx.has_bias else None), None, None,
                None)


def layer_norm_with_skip(x, weight, bias, eps: float = 1e-5):
    """``(layer_norm(x), x)`` where the second output carries the skip connection (see ``_LayerNormFn``)."""
    if use_native(x) and x.dtype in (torch.bfloat16, torch.float32) and weight is not None and x.requires_grad:
        if _graph_node(x, weight, bias):
            return load_ext().norm_skip_node(x, weight, bias, eps, False)
        return _call(_LayerNormFn, x, weight, bias, eps, False, True)
    return layer_norm(x, weight, bias, eps), x


def layer_norm(x, weight, bias, eps: float = 1e-5):
    if use_native(x) and x.dtype in (torch.bfloat16, torch.float32) and weight is not None:
        if _graph_node(x, weight, bias):
            return load_ext().norm_node(x, weight, bias, eps, False)
        return _call(_LayerNormFn, x, weight, bias, eps, False)
    w = None if weight is None else weight.float()
    b = None if bias is None else bias.float()
    return F.layer_norm(x.float(), (x.shape[-1],), w, b, eps).to(x.dtype)


def rms_norm_with_skip(x, weight, eps: float = 1e-6):
    """``(rms_norm(x), x)``; the gradient of the second output is added inside the norm's backward kernel (see ``_LayerNormFn``)."""
    if use_native(x) and x.dtype in (torch.bfloat16, torch.float32) and x.requires_grad:
        if _graph_node(x, weight):
            return load_ext().norm_skip_node(x, weight, None, eps, True)
        return _call(_LayerNormFn, x, weight, None, eps, True, True)
    return rms_norm(x, weight, eps), x


def rms_norm(x, weight, eps: float = 1e-6):
    if use_native(x) and x.dtype in (torch.bfloat16, torch.float32):
        if _graph_node(x, weight):
            return load_ext().norm_node(x, weight, None, eps, True)
        return _call(_LayerNormFn, x, weight, None, eps, True)
    xf = x.float()
    y = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps)
    return (y * weight.float()).to(x.dtype)


# --------------------------------------------------------------------------------------
# bias + gelu, bias + dropout + residual
# --------------------------------------------------------------------------------------
class _BiasActFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, bias, act):
        ext = load_ext()
        x2 = x.reshape(-1, x.shape[-1]).contiguous()
        y = ext.bias_act_fwd(x2, bias, _ACT_IDS[act])
        count_launch()
        ctx.save_for_backward(x2, bias)
        ctx.act = act
        ctx.bias_param = bias
        return y.view(x.shape)

    @staticmethod
    def backward(ctx, gy):
        ext = load_ext()
        x2, bias = ctx.saved_tensors
        g2 = gy.reshape(-1, gy.shape[-1]).contiguous()
        gx = ext.bias_act_bwd(g2, x2, bias, _ACT_IDS[ctx.act])
        count_launch()
        gb = None
        if bias is not None and ctx.needs_input_grad[1]:
            gb = _bias_grad(ext, gx, ctx.bias_param)
        return gx.view(gy.shape), gb, None


def bias_act(x, bias, act: str = "gelu"):
    """``act(x + bias)`` (replaces ``fused_bias_add_gelu``)."""
    if use_native(x) and x.dtype == torch.bfloat16:
        return _call(_BiasActFn, x, bias, act)
    y = x if bias is None else x + bias.to(x.dtype)
    return _act_ref(y, act)


def bias_gelu(x, bias):
    return bias_act(x, bias, "gelu")


def tp_rng_salt(sharded: bool) -> int:
    """Salt of the dropout RNG stream (tensor-parallel aware).  All tensor-parallel ranks of a model replica share
    one (seed, offset) sequence (``dutil.model_parallel_seed``); activations that are *sharded* over the TP group
    (attention heads, token shards under sequence parallelism) must see different masks on different ranks → the TP
    rank is mixed into the Philox key; *replicated* activations (salt 0) get identical masks everywhere."""
    if not sharded:
        return 0
    from libai_b200.utils import distributed as dutil

    topo = dutil.get_dist_util()
    return topo.tp_rank + 1 if topo.tensor_parallel_size > 1 else 0


def _activations_token_sharded() -> bool:
    from libai_b200.utils import distributed as dutil

    return bool(dutil.get_dist_util().sequence_parallel)


class _BiasDropoutAddFn(torch.autograd.Function):
    """``residual + dropout(x + bias)`` in one native kernel; the mask is a pure function of the Philox
    ``(seed, offset)`` pair stored by the forward and the element index, so nothing but 16 bytes is kept for backward."""

    @staticmethod
    def forward(ctx, x, bias, residual, p, salt):
        ext = load_ext()
        x2 = x.reshape(-1, x.shape[-1]).contiguous()
        r2 = None if residual is None else residual.reshape(-1, x.shape[-1]).contiguous()
        y, rng_state = ext.bias_dropout_residual(x2, bias, r2, p, salt, None)
        count_launch()
        ctx.save_for_backward(rng_state)
        ctx.p, ctx.bias_param, ctx.has_res = p, bias, residual is not None
        return y.view(x.shape)

    @staticmethod
    def backward(ctx, gy):
        ext = load_ext()
        (rng_state,) = ctx.saved_tensors
        g2 = gy.reshape(-1, gy.shape[-1]).contiguous()
        gx, _ = ext.bias_dropout_residual(g2, None, None, ctx.p, 0, rng_state)
        count_launch()
        gb = None
        if ctx.bias_param is not None and ctx.needs_input_grad[1]:
            gb = _bias_grad(ext, gx, ctx.bias_param)
        return gx.view(gy.shape), gb, (gy if ctx.has_res else None), None, None


def bias_dropout_add(x, bias, residual, p: float, training: bool, sharded=None):
    """``residual + dropout(x + bias)`` (replaces ``fused_bias_add_dropout`` + the add).  ``sharded``: whether ``x`` is
    sharded over the tensor-parallel group (default: yes iff sequence parallelism is on), see :func:`tp_rng_salt`."""
    if use_native(x) and x.dtype == torch.bfloat16 and x.shape[-1] % 8 == 0:
        if p == 0.0 or not training:
            return _call(_BiasAddFn, x, bias, residual)
        if sharded is None:
            sharded = _activations_token_sharded()
        return _call(_BiasDropoutAddFn, x, bias, residual, float(p), tp_rng_salt(sharded))
    y = x if bias is None else x + bias.to(x.dtype)
    y = F.dropout(y, p=p, training=training)
    return y if residual is None else residual + y


def dropout(x, p: float, training: bool, sharded: bool = False):
    """Native Philox dropout (same kernel as :func:`bias_dropout_add` without bias / residual)."""
    if p == 0.0 or not training:
        return x
    if use_native(x) and x.dtype == torch.bfloat16 and x.shape[-1] % 8 == 0:
        return _call(_BiasDropoutAddFn, x, None, None, float(p), tp_rng_salt(sharded))
    return F.dropout(x, p=p, training=training)


class _BiasAddFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, bias, residual):
        ext = load_ext()
        x2 = x.reshape(-1, x.shape[-1]).contiguous()
        r2 = None if residual is None else residual.reshape(-1, x.shape[-1]).contiguous()
        y = ext.bias_residual_fwd(x2, bias, r2)
        count_launch()
        ctx.has_bias = bias is not None
        ctx.bias_param = bias
        ctx.has_res = residual is not None
        return y.view(x.shape)

    @staticmethod
    def backward(ctx, gy):
        gb = None
        if ctx.has_bias and ctx.needs_input_grad[1]:
            gb = _bias_grad(load_ext(), gy.reshape(-1, gy.shape[-1]).contiguous(), ctx.bias_param)
        return gy, gb, (gy if ctx.has_res else None)


# --------------------------------------------------------------------------------------
# attention
# --------------------------------------------------------------------------------------
def attention_ref(q, k, v, *, causal: bool, scale: float, mask=None, bias=None, dropout_p: float = 0.0,
                  training: bool = False, fill: float = -10000.0):
    """Unfused attention on ``[b, a, s, d]`` tensors. ``mask``: 1 = keep, 0 = masked
    (filled with ``fill`` like the reference: libai/layers/attention.py:223-245)."""
    scores = torch.matmul(q.float(), k.float().transpose(-1, -2)) * scale
    if bias is not None:
        scores = scores + bias.float()
    sq, sk = scores.shape[-2], scores.shape[-1]
    if causal:
        tril = torch.ones(sq, sk, dtype=torch.bool, device=q.device).tril(diagonal=sk - sq)
        scores = torch.where(tril, scores, torch.full_like(scores, fill))
    if mask is not None:
        scores = torch.where(mask.bool(), scores, torch.full_like(scores, fill))
    probs = torch.softmax(scores, dim=-1)
    probs = F.dropout(probs, p=dropout_p, training=training)
    return torch.matmul(probs, v.float()).to(q.dtype)


def _prep_bias(bias, q):
    """Additive score bias for the flash kernel: bf16 ``[B|1, A|1, S, S]`` with contiguous keys."""
    if bias is None:
        return None
    b = bias
    while b.dim() < 4:
        b = b.unsqueeze(0)
    if b.dtype != torch.bfloat16:
        b = b.to(torch.bfloat16)
    if b.stride(-1) != 1 or b.stride(-2) % 8 or b.stride(0) % 8 or b.stride(1) % 8 or b.data_ptr() % 16:
        b = b.contiguous()
    return b


class _FlashAttnFn(torch.autograd.Function):
    """Flash attention on ``[b, a, s, d]`` views with optional additive bias (dense or ALiBi slopes), key-padding
    lengths and Philox dropout on the probabilities — all inside the tcgen05 kernels."""

    @staticmethod
    def forward(ctx, q, k, v, causal, scale, bias, alibi_slopes, p_drop, kv_lens):
        ext = load_ext()
        b = _prep_bias(bias, q)
        o, lse, rng_state = ext.attn_fwd(q, k, v, causal, scale, kv_lens, b, alibi_slopes, p_drop,
                                         tp_rng_salt(True) if p_drop > 0 else 0)
        count_launch()
        ctx.save_for_backward(q, k, v, o, lse, b, alibi_slopes, rng_state, kv_lens)
        ctx.causal, ctx.scale, ctx.p_drop = causal, scale, p_drop
        ctx.bias_shape = None if bias is None else (bias.shape, bias.dtype)
        return o

    @staticmethod
    def backward(ctx, go):
        ext = load_ext()
        q, k, v, o, lse, b, slopes, rng_state, kv_lens = ctx.saved_tensors
        dbias = None
        if b is not None and ctx.needs_input_grad[5]:
            dbias = torch.zeros(b.shape, dtype=torch.float32, device=b.device)
            if dbias.stride() != b.stride():
                dbias = torch.empty_strided(b.shape, b.stride(), dtype=torch.float32, device=b.device).zero_()
        dq, dk, dv, _ = ext.attn_bwd(go, q, k, v, o, lse, ctx.causal, ctx.scale, kv_lens, b, slopes, dbias, ctx.p_drop,
                                     rng_state if ctx.p_drop > 0 else None)
        count_launch(3)
        gb = None
        if dbias is not None:
            shape, dtype = ctx.bias_shape
            gb = dbias.to(dtype).reshape(shape)
        return dq, dk, dv, None, None, gb, None, None, None


class _FlashAttnPackedFn(torch.autograd.Function):
    """Self-attention straight from the packed QKV projection ``[b, s, a, 3d]`` (per-head ``[q|k|v]``):
    the kernels read q/k/v through strided TMA maps and the backward writes one packed ``dqkv`` – no
    slicing, no gradient accumulation kernels around the attention."""

    @staticmethod
    def forward(ctx, qkv, causal, scale, kv_lens, p_drop=0.0, alibi_slopes=None):
        ext = load_ext()
        d = qkv.shape[-1] // 3
        v4 = qkv.permute(0, 2, 1, 3)
        q, k, v = v4[..., :d], v4[..., d : 2 * d], v4[..., 2 * d :]
        o, lse, rng_state = ext.attn_fwd(q, k, v, causal, scale, kv_lens, None, alibi_slopes, p_drop,
                                         tp_rng_salt(True) if p_drop > 0 else 0)
        count_launch()
        ctx.save_for_backward(qkv, o, lse, kv_lens, rng_state, alibi_slopes)
        ctx.causal, ctx.scale, ctx.p_drop = causal, scale, p_drop
        return o.permute(0, 2, 1, 3)  # [b, s, a, d] contiguous

    @staticmethod
    def backward(ctx, go):
        ext = load_ext()
        qkv, o, lse, kv_lens, rng_state, slopes = ctx.saved_tensors
        d = qkv.shape[-1] // 3
        v4 = qkv.permute(0, 2, 1, 3)
        q, k, v = v4[..., :d], v4[..., d : 2 * d], v4[..., 2 * d :]
        _, _, _, dqkv = ext.attn_bwd(go.permute(0, 2, 1, 3), q, k, v, o, lse, ctx.causal, ctx.scale, kv_lens, None, slopes,
                                     None, ctx.p_drop, rng_state if ctx.p_drop > 0 else None)
        count_launch(3)
        return dqkv.view(qkv.shape), None, None, None, None, None


# ---- attention with 32-bit probabilities (csrc/attention_split_sm100.cu) ----------------------------------------------
def _rows_of_vectors(t) -> bool:
    """A view whose rows TMA can read: contiguous last dimension, every other stride and the base on 16 bytes."""
    return t.data_ptr() % 16 == 0 and t.stride(-1) == 1 and all(n == 1 or (st > 0 and st % 8 == 0) for n, st in zip(t.shape[:-1], t.stride()))


def _split_views(layout: str, ts):
    """``[b, a, s, d]`` views of q, k, v; ``qkv``: packed ``[b, s, a, 3d]``, ``q_kv``: ``[b, s, a, d]`` and ``[b, sk, a, 2d]``."""
    if layout == "qkv":
        return ts[0].permute(0, 2, 1, 3).chunk(3, -1)
    if layout == "q_kv":
        return (ts[0].permute(0, 2, 1, 3), *ts[1].permute(0, 2, 1, 3).chunk(2, -1))
    return ts


def _mask_supported(mask, q_sizes, device, sk: int) -> bool:
    """``q_sizes``: ``(b, a, sq)``."""
    return (mask.device == device and not mask.is_complex() and mask.dim() <= 4
            and all(m in (1, n) for m, n in zip(reversed(mask.shape), (sk, q_sizes[2], q_sizes[1], q_sizes[0]))))


def _pack_mask(ext, mask, q, sk: int, causal: bool):
    m = mask[(None,) * (4 - mask.dim())]
    count_launch()
    return ext.attn_mask_pack(m.expand(m.shape[0], m.shape[1], q.shape[2], sk), causal)


def _split_sizes_ok(b, a, sq, sk, d, scale, causal) -> bool:
    return (d % 8 == 0 and 8 <= d <= 64 and min(b, a, sq, sk) > 0 and max(a, b) <= 65535 and scale > 0 and (not causal or sk >= sq))


def _split_supported(q, k, v, scale, causal, mask) -> bool:
    """Sizes and types of the kernels with 32-bit probabilities, from ``[b, a, s, d]`` views.  Other head dims stay with the flash
    kernels (64 / 128 without a mask: bf16 probabilities, as ever) or with the unfused form."""
    return (use_native(q) and q.dtype == k.dtype == v.dtype == torch.bfloat16 and q.device == k.device == v.device
            and q.dim() == k.dim() == 4 and k.shape == v.shape and q.shape[:2] == k.shape[:2] and q.shape[-1] == k.shape[-1]
            and _split_sizes_ok(*q.shape[:3], k.shape[2], q.shape[3], scale, causal)
            and (mask is None or _mask_supported(mask, q.shape[:3], q.device, k.shape[2])) and type(q) is not FakeTensor and _plain_call())


def _split_graph_backward(go, layout: str, causal: bool, scale: float, mask, ts, needed) -> list:
    """Gradients of ``ts`` with a graph of their own: the unfused form is differentiated."""
    out = attention_ref(*_split_views(layout, ts), causal=causal, scale=scale, mask=mask)
    out = out if layout == "q_k_v" else out.permute(0, 2, 1, 3)
    grads = iter(torch.autograd.grad(out, [t for t, n in zip(ts, needed) if n], go, create_graph=True))
    return [next(grads) if n else None for n in needed]


_SPLIT_LAYOUTS = {"qkv": 0, "q_kv": 1, "q_k_v": 2}


class _SplitAttnFn(torch.autograd.Function):
    """Attention whose probabilities reach the tensor core as three bf16 parts (``layout``: see :func:`_split_views`)."""

    @staticmethod
    def forward(ctx, layout, causal, scale, mask, *ts):
        ext = load_ext()
        q, k, v = _split_views(layout, ts)
        words, fill = (None, None) if mask is None else _pack_mask(ext, mask, q, k.shape[2], causal)
        train = any(ctx.needs_input_grad[4:])
        o, o32, lse = ext.attn_split_fwd(q, k, v, causal and mask is None, scale, words, fill, train)
        count_launch()
        out = o if layout == "q_k_v" else o.permute(0, 2, 1, 3)
        if train:
            ctx.save_for_backward(o32, lse, words, fill, *ts)
            ctx.layout, ctx.causal, ctx.scale, ctx.mask = layout, causal, scale, mask
        return out

    @staticmethod
    def backward(ctx, go):
        o32, lse, words, fill, *ts = ctx.saved_tensors
        q, k, v = _split_views(ctx.layout, ts)
        if torch.is_grad_enabled():
            return (None,) * 4 + tuple(_split_graph_backward(go, ctx.layout, ctx.causal, ctx.scale, ctx.mask, ts, ctx.needs_input_grad[4:]))
        if ctx.layout == "q_k_v":              # gradients backed by [b, s, a, d], as the projections around an attention read them
            gs = [torch.empty(t.shape[0], t.shape[2], t.shape[1], t.shape[3], dtype=t.dtype, device=t.device).permute(0, 2, 1, 3) for t in ts]
        else:
            gs = [torch.empty(t.shape, dtype=t.dtype, device=t.device) for t in ts]
            go = go.permute(0, 2, 1, 3)
        load_ext().attn_split_bwd(go, q, k, v, o32, lse, *_split_views(ctx.layout, gs), ctx.causal and words is None, ctx.scale, words, fill)
        count_launch(3)
        return (None,) * 4 + tuple(gs)


def attention_packed(layout: str, ts, *, causal: bool, scale: float, mask=None, dropout_p: float = 0.0, training: bool = False):
    """Attention straight from packed projections, ``qkv`` ``([b, s, a, 3d],)`` or ``q_kv`` ``([b, s, a, d], [b, sk, a, 2d])``, with an
    optional dense 0/1 mask, → ``[b, s, a, d]``; ``None`` where the kernels do not apply (the caller slices and takes :func:`attention`)."""
    x, y = ts[0], ts[-1]
    b, sq, a, d = x.shape
    d = d // 3 if layout == "qkv" else d
    if ((dropout_p > 0.0 and training) or not use_native(x) or type(x) is FakeTensor or not _plain_call() or not _split_sizes_ok(b, a, sq, y.shape[1], d, scale, causal)
            or any(t.dtype != torch.bfloat16 or t.device != x.device or not t.is_contiguous() or t.data_ptr() % 16 for t in ts)
            or (layout == "q_kv" and y.shape != (b, y.shape[1], a, 2 * d)) or (layout == "qkv" and x.shape[3] != 3 * d)
            or (mask is not None and not _mask_supported(mask, (b, a, sq), x.device, y.shape[1]))):
        return None
    if _graph_node(mask, *ts):
        return load_ext().split_attention_node(list(ts), causal, float(scale), mask, _SPLIT_LAYOUTS[layout])
    return _call(_SplitAttnFn, layout, causal, float(scale), mask, *ts)


def _cache_too_long_for_one_cluster(heads: int, keys: int, d: int) -> bool:
    """A head's keys are read by at most eight CTAs, in steps of 1.05 us (128 threads, ``lanes`` per key, four keys each); copies and products
    over the whole chip take 28 us and 1.2e-5 us per number of the caches.  So up to three heads in all with a very long past stay with
    those: 1 head x 100000 x 128 496 against 154 us, 2 x 32768 x 64 68 against 88, 4 x 4096 x 128 21 against 39, 8 x 32768 x 128 198 against 335."""
    if heads > 3:
        return False
    lanes = 1 << (d // 8 - 1).bit_length()
    return 5.0 + 1.05 * keys / (8 * 512 / lanes) > 28.0 + 1.2e-5 * heads * keys * d


def attention_cached(q, k_new, v_new, past_key, past_value, *, scale: float, mask=None, dropout_p: float = 0.0, training: bool = False):
    """One new token per sequence: ``q``, ``k_new``, ``v_new`` ``[b, a, 1, d]``, the caches ``[b, a, past, d]`` → (context
    ``[b, 1, a, d]``, the caches with the token appended) in one kernel; ``None`` where it does not apply (gradients, several new
    tokens, other types, caches held on another device, a very long past of up to three heads): the caller concatenates and takes :func:`attention`."""
    if not use_native(q) or type(q) is FakeTensor or not _plain_call() or q.dim() != 4 or past_key.dim() != 4:
        return None
    ts, qs, ps = (q, k_new, v_new, past_key, past_value), q.shape, past_key.shape
    b, a, new, d = qs
    if (new != 1 or (dropout_p > 0.0 and training) or scale <= 0
            or not torch.bfloat16 == q.dtype == k_new.dtype == v_new.dtype == past_key.dtype == past_value.dtype
            or not q.device == k_new.device == v_new.device == past_key.device == past_value.device or not qs == k_new.shape == v_new.shape
            or ps != past_value.shape or ps[:2] != qs[:2] or ps[3] != d or ps[2] == 0 or min(b, a, d) == 0 or max(b, a) > 65535 or d % 8 or d > 256
            or not all(_rows_of_vectors(t) for t in ts) or (torch.is_grad_enabled() and any(t.requires_grad for t in ts))
            or (mask is not None and not _mask_supported(mask, qs[:3], q.device, ps[2] + 1))
            or (b * a < 4 and _cache_too_long_for_one_cluster(b * a, ps[2], d))):
        return None
    ext = load_ext()
    words, fill = (None, None) if mask is None else _pack_mask(ext, mask, q, ps[2] + 1, False)
    count_launch()
    return ext.attn_decode(q, k_new, v_new, past_key, past_value, float(scale), words, fill)


def attention_qkvpacked_supported(qkv, mask, dropout_p, training) -> bool:
    return (
        use_native(qkv)
        and qkv.dtype == torch.bfloat16
        and mask is None
        and qkv.shape[-1] // 3 in (64, 128)
        and qkv.is_contiguous()
    )


def attention_qkvpacked(qkv, *, causal: bool, scale: float, kv_lens=None, dropout_p: float = 0.0, training: bool = False,
                        alibi_slopes=None):
    """qkv ``[b, s, a, 3d]`` → context ``[b, s, a, d]``; ``kv_lens`` (int32 ``[b]``): valid keys per sample
    of a right-padded batch (keys beyond it are masked inside the kernel); ``dropout_p`` > 0 in training drops
    attention probabilities inside the kernel (Philox, TP-rank salted)."""
    p = float(dropout_p) if training else 0.0
    if _graph_node(qkv, kv_lens, alibi_slopes):
        return load_ext().flash_packed_node(qkv, causal, float(scale), kv_lens, p, alibi_slopes, tp_rng_salt(True) if p > 0 else 0)
    return _call(_FlashAttnPackedFn, qkv, causal, float(scale), kv_lens, p, alibi_slopes)


def attention(q, k, v, *, causal: bool = False, scale: Optional[float] = None, mask=None, bias=None,
              dropout_p: float = 0.0, training: bool = False, alibi_slopes=None, kv_lens=None):
    """Softmax attention on ``[b, a, s, d]``.  The native flash kernels handle causal / full / key-padding
    (``kv_lens``) masking, an additive score bias (dense ``[b|1, a|1, s, s]`` — T5 relative positions — or
    ``alibi_slopes`` ``[a]``) and dropout on the probabilities.  Dense 0/1 masks, query and key lengths of their own and the
    head dims below 64 run in the kernels with 32-bit probabilities; what is left (dropout or bias beside those, head dims
    above 64 beside those) uses the unfused form."""
    if scale is None:
        scale = 1.0 / math.sqrt(q.shape[-1])
    if (
        use_native(q)
        and q.dtype == torch.bfloat16
        and mask is None
        and q.shape[-1] in (64, 128)
        and q.shape[-2] == k.shape[-2]
        and q.shape[-2] % 8 == 0
        and (bias is None or (bias.shape[-1] == k.shape[-2] and bias.shape[-2] == q.shape[-2]))
    ):
        # strided [b, a, s, d] views of the packed QKV projection are consumed directly (TMA strides)
        return _call(_FlashAttnFn, q, k, v, causal, float(scale), bias, alibi_slopes, float(dropout_p) if training else 0.0, kv_lens)
    if (bias is None and alibi_slopes is None and kv_lens is None and not (dropout_p > 0.0 and training)
            and _split_supported(q, k, v, scale, causal, mask)):
        ts = [t if _rows_of_vectors(t) else t.contiguous() for t in (q, k, v)]
        if all(_rows_of_vectors(t) for t in ts):
            if _graph_node(mask, *ts):
                return load_ext().split_attention_node(ts, causal, float(scale), mask, 2)
            return _call(_SplitAttnFn, "q_k_v", causal, float(scale), mask, *ts)
    if alibi_slopes is not None:
        sq, sk = q.shape[-2], k.shape[-2]
        rel = torch.arange(sk, device=q.device)[None, :] - torch.arange(sk - sq, sk, device=q.device)[:, None]
        ab = alibi_slopes.float()[None, :, None, None] * rel[None, None].float()
        bias = ab if bias is None else bias.float() + ab
    return attention_ref(q, k, v, causal=causal, scale=scale, mask=mask, bias=bias,
                         dropout_p=dropout_p, training=training)


# --------------------------------------------------------------------------------------
# vocab-parallel softmax cross entropy
# --------------------------------------------------------------------------------------
class _VocabParallelCE(torch.autograd.Function):
    """Per-token CE over logits whose last dim is split across ``group``.

    fwd: local (max, sum-exp, target-logit) → 3 tiny all-reduces → loss; bwd: softmax − onehot
    written in place of the saved logits (no extra ``[T, V/t]`` buffer)."""

    @staticmethod
    def forward(ctx, logits, labels, vocab_start, group):
        T, Vl = logits.shape
        world = 1 if group is None else dist.get_world_size(group)
        native = use_native(logits) and logits.dtype in (torch.bfloat16, torch.float32)
        if native:
            ext = load_ext()
            mx, se, tgt = ext.ce_stats(logits, labels, vocab_start)
            count_launch()
        else:
            lf = logits.float()
            mx = lf.max(dim=-1).values
            se = torch.exp(lf - mx[:, None]).sum(-1)
            local = labels - vocab_start
            inside = (local >= 0) & (local < Vl)
            idx = local.clamp(0, Vl - 1)
            tgt = torch.where(inside, lf.gather(1, idx[:, None]).squeeze(1), torch.zeros_like(mx))
        if world > 1:
            gmx = mx.clone()
            dist.all_reduce(gmx, op=dist.ReduceOp.MAX, group=group)
            se = se * torch.exp(mx - gmx)
            packed = torch.stack([se, tgt])
            dist.all_reduce(packed, group=group)
            se, tgt = packed[0], packed[1]
            mx = gmx
        lse = mx + torch.log(se)
        loss = lse - tgt
        ctx.save_for_backward(logits, labels, lse)
        ctx.vocab_start = vocab_start
        ctx.native = native
        return loss

    @staticmethod
    def backward(ctx, gloss):
        logits, labels, lse = ctx.saved_tensors
        if ctx.native:
            ext = load_ext()
            g = ext.ce_bwd(logits, labels, lse, gloss.contiguous().float(), ctx.vocab_start)
            count_launch()
            return g, None, None, None
        Vl = logits.shape[1]
        p = torch.exp(logits.float() - lse[:, None])
        local = labels - ctx.vocab_start
        inside = (local >= 0) & (local < Vl)
        idx = local.clamp(0, Vl - 1)
        p.scatter_add_(1, idx[:, None], -inside.to(p.dtype)[:, None])
        return (p * gloss.float()[:, None]).to(logits.dtype), None, None, None


def vocab_parallel_cross_entropy(logits, labels, vocab_start: int = 0, group=None):
    """logits ``[..., V/t]``, labels ``[...]`` (global ids) → per-token loss ``[...]`` (fp32)."""
    shp = labels.shape
    rows, flat = logits.reshape(-1, logits.shape[-1]), labels.reshape(-1)
    if (_graph_node(logits, labels) and (group is None or dist.get_world_size(group) == 1) and use_native(logits)
            and logits.dtype in (torch.bfloat16, torch.float32)):
        return load_ext().cross_entropy_node(rows, flat, int(vocab_start)).view(shp)
    return _call(_VocabParallelCE, rows, flat, vocab_start, group).view(shp)


# --------------------------------------------------------------------------------------
# embedding
# --------------------------------------------------------------------------------------
class _EmbeddingFn(torch.autograd.Function):
    """Row gather; the backward scatters ``gy`` straight into the table's fp32 ``main_grad`` with vector reductions
    (no sort / segment-reduce / temporary gradient the size of the table, and no later fold of ``p.grad``)."""

    @staticmethod
    def forward(ctx, ids, table, vocab_start):
        ext = load_ext()
        flat = ids.reshape(-1).contiguous()
        out = ext.embedding_fwd(flat, table, vocab_start)
        count_launch()
        ctx.save_for_backward(flat)
        ctx.table = table
        ctx.vocab_start = vocab_start
        return out.view(*ids.shape, table.shape[1])

    @staticmethod
    def backward(ctx, gy):
        (flat,) = ctx.saved_tensors
        table = ctx.table
        g2 = gy.reshape(-1, gy.shape[-1]).contiguous()
        ext = load_ext()
        count_launch()
        main_grad = getattr(table, "main_grad", None)
        if main_grad is not None and main_grad.dtype == torch.float32:
            ext.embedding_bwd(flat, g2, main_grad, ctx.vocab_start)
            table.grad_added_to_main_grad = True
            return None, None, None
        grad = torch.zeros(table.shape, dtype=torch.float32, device=table.device)
        ext.embedding_bwd(flat, g2, grad, ctx.vocab_start)
        return None, grad.to(table.dtype), None


def embedding(ids, table, vocab_start: int = 0):
    """Row gather with zero rows for ids outside ``[vocab_start, vocab_start + rows)``."""
    rows = table.shape[0]
    if (use_native(table) and table.dtype == torch.bfloat16 and table.dim() == 2 and table.shape[1] % 8 == 0
            and table.is_contiguous() and ids.dtype == torch.long):
        return _call(_EmbeddingFn, ids, table, int(vocab_start))
    local = ids - vocab_start
    inside = (local >= 0) & (local < rows)
    out = F.embedding(local.clamp(0, rows - 1), table)
    return out * inside.unsqueeze(-1).to(out.dtype)


# --------------------------------------------------------------------------------------
# rotary position embedding
# --------------------------------------------------------------------------------------
def rotate_half(x):
    x1, x2 = x[..., : x.shape[-1] // 2], x[..., x.shape[-1] // 2 :]
    return torch.cat((-x2, x1), dim=-1)


class _RopeFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, cos, sin):
        ext = load_ext()
        ctx.save_for_backward(cos, sin)
        count_launch()
        return ext.rope(x.contiguous(), cos, sin, False)

    @staticmethod
    def backward(ctx, g):
        ext = load_ext()
        cos, sin = ctx.saved_tensors
        count_launch()
        return ext.rope(g.contiguous(), cos, sin, True), None, None


def apply_rotary(x, cos, sin):
    """x ``[b, a, s, d]``; cos/sin ``[s, d]`` (HF "rotate_half" convention; reference
    projects/Llama/llama.py:31-43)."""
    if use_native(x) and x.dtype == torch.bfloat16 and cos.dtype == torch.float32:
        return _call(_RopeFn, x, cos, sin)
    c = cos[None, None].to(x.dtype)
    s = sin[None, None].to(x.dtype)
    return x * c + rotate_half(x) * s



class _RopeQKVFn(torch.autograd.Function):
    """Rotary embedding on q and k of the packed projection ``[b, s, a, 3d]`` in one pass (v copied);
    the backward rotates the packed ``dqkv`` of the attention kernel in place with the inverse rotation."""

    @staticmethod
    def forward(ctx, qkv, cos, sin, pos_offset):
        ext = load_ext()
        ctx.save_for_backward(cos, sin)
        ctx.pos_offset = pos_offset
        count_launch()
        return ext.rope_qkv(qkv, cos, sin, pos_offset, False, False)

    @staticmethod
    def backward(ctx, g):
        ext = load_ext()
        cos, sin = ctx.saved_tensors
        count_launch()
        g = g if g.is_contiguous() else g.contiguous()
        return ext.rope_qkv(g, cos, sin, ctx.pos_offset, True, True), None, None, None


def apply_rotary_qkv(qkv, cos, sin, pos_offset: int = 0):
    """qkv ``[b, s, a, 3d]`` (per-head ``[q|k|v]``); cos/sin fp32 ``[max_pos, d]``; token ``i`` of the
    sequence uses position ``i + pos_offset``."""
    if use_native(qkv) and qkv.dtype == torch.bfloat16 and cos.dtype == torch.float32 and qkv.is_contiguous():
        if _graph_node(qkv, cos, sin):
            return load_ext().rope_qkv_node(qkv, cos, sin, int(pos_offset))
        return _call(_RopeQKVFn, qkv, cos, sin, int(pos_offset))
    d = qkv.shape[-1] // 3
    s_len = qkv.shape[1]
    c = cos[pos_offset : pos_offset + s_len, None, :].to(qkv.dtype)
    sn = sin[pos_offset : pos_offset + s_len, None, :].to(qkv.dtype)
    q, k, v = qkv[..., :d], qkv[..., d : 2 * d], qkv[..., 2 * d :]
    return torch.cat([q * c + rotate_half(q) * sn, k * c + rotate_half(k) * sn, v], dim=-1)


# --------------------------------------------------------------------------------------
# fused softmax variants kept for exact-parity tests
# --------------------------------------------------------------------------------------
def fused_scale_mask_softmax(scores, mask=None, scale: float = 1.0, causal: bool = False, fill: float = -10000.0):
    s = scores.float() * scale
    if causal:
        sq, sk = s.shape[-2:]
        tril = torch.ones(sq, sk, dtype=torch.bool, device=s.device).tril(diagonal=sk - sq)
        s = torch.where(tril, s, torch.full_like(s, fill))
    if mask is not None:
        s = torch.where(mask.bool(), s, torch.full_like(s, fill))
    return torch.softmax(s, dim=-1).to(scores.dtype)


def swiglu(gate, up):
    """``silu(gate) * up`` (reference projects/Llama/llama.py:111-113)."""
    if use_native(gate) and gate.dtype == torch.bfloat16:
        return _call(_SwigluFn, gate, up)
    return F.silu(gate) * up


class _SwigluFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, gate, up):
        ext = load_ext()
        g, u = gate.contiguous(), up.contiguous()
        ctx.save_for_backward(g, u)
        count_launch()
        return ext.swiglu_fwd(g, u)

    @staticmethod
    def backward(ctx, gy):
        ext = load_ext()
        g, u = ctx.saved_tensors
        count_launch()
        dg, du = ext.swiglu_bwd(gy.contiguous(), g, u)
        return dg, du
