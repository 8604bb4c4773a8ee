"""Autograd bindings of the hand-written sm_100a kernels.

Each op launches the kernels of ``csrc/kernels`` on the current CUDA stream, forward and
backward.  The ops a block is made of are C++ autograd nodes (``csrc/torch``): issued from
Python they left the device idle for half of a small layer's time.  There is no eager
fallback here: if a native library is missing these raise.
"""
from __future__ import annotations

import os
import threading
from typing import Optional

import torch

from .native import cuda_lib, dtype_code, ptr, stream_handle, torch_ops


def _check(rc: int, what: str):
    if rc != 0:
        raise RuntimeError(f"{what} failed (code {rc})")


# --------------------------------------------------------------------- GEMM
WORKSPACE_WANTED = -5                                # gemm_tcgen05.cu, kWorkspaceWanted


def gemm(a: torch.Tensor, a_mn: bool, b: torch.Tensor, b_mn: bool, m: int, n: int, k: int,
         out: Optional[torch.Tensor] = None, accumulate: bool = False,
         out_dtype: Optional[torch.dtype] = None, add: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``out[m, n] (+)= sum_k A(m, k) B(n, k)`` on the tcgen05 tensor cores.
    ``a`` is stored ``[m, k]`` (``a_mn=False``) or ``[k, m]`` (``a_mn=True``);
    ``b`` is stored ``[n, k]`` or ``[k, n]`` likewise.  Inputs are 2-D with unit
    inner stride.  ``add`` (``[m, n]``, the type of ``out``, unit inner stride) is added
    to the product in the epilogue: ``out = A B^T + add``."""
    if a.dtype != b.dtype or a.dtype not in (torch.bfloat16, torch.float16):
        raise TypeError("gemm operands must both be bf16 or both fp16")
    if a.stride(-1) != 1 or b.stride(-1) != 1:
        raise ValueError("gemm operands need unit inner stride")
    if out is None:
        out = torch.empty(m, n, dtype=out_dtype or a.dtype, device=a.device)
        accumulate = False
    if add is not None:
        if add.shape != (m, n) or add.dtype != out.dtype or add.stride(-1) != 1:
            raise ValueError("gemm: `add` must be [m, n] of the output's type with unit inner stride")
    lib, c_dtype = cuda_lib(), dtype_code(out.dtype)
    args = (ptr(a), a_mn, a.stride(0), ptr(b), b_mn, b.stride(0), ptr(out), out.stride(0), c_dtype, accumulate)
    rest = (m, n, k, dtype_code(a.dtype))
    if add is None:
        rc = lib.ft_gemm_try(*args, *rest, stream_handle())
        args += (None, 0, None, *rest)
    else:
        args += (ptr(add), add.stride(0), None, *rest)
        rc = lib.ft_gemm_ws(*args, None, -1, stream_handle())
    if rc == WORKSPACE_WANTED:                       # the product is divided along k, with scratch for partial sums
        nbytes = lib.ft_gemm_ws_bytes(m, n, k, c_dtype)
        try:
            ws = torch.empty(nbytes, dtype=torch.uint8, device=a.device)
        except torch.OutOfMemoryError:               # it runs whole then
            ws, nbytes = None, 0
        rc = lib.ft_gemm_ws(*args, ptr(ws), nbytes, stream_handle())
    _check(rc, "ft_gemm" if add is None else "ft_gemm_add")
    return out


def _gathered_product(x, w):
    """``x w^T`` of a weight whose rows other ranks own are not in the gathered buffer yet: one
    kernel brings them in over NVLink and multiplies (csrc/comm/ag_gemm.cu).  None where that kernel
    does not cover the shape; the weight is complete then."""
    pending, k = w._ft_gather, x.shape[-1]
    with torch.no_grad():
        x2 = x.reshape(-1, k)
        if x2.stride(-1) != 1 or (x2.stride(0) * x2.element_size()) % 16:
            x2 = x2.contiguous()
        if not pending.covers(x2.shape[0], k):
            pending.complete_without_product()
            return None
        y = torch.empty(*x.shape[:-1], w.shape[0], dtype=x.dtype, device=x.device)
        pending.run(x2, y.view(-1, w.shape[0]))
        return y


def linear(x, w):
    done = _gathered_product(x, w) if getattr(w, "_ft_gather", None) is not None else None
    return torch_ops().linear(x, w, None, None, done)


def linear_add(x, w, res):
    """``res + x w^T`` with the addition in the GEMM epilogue (one read of ``res`` instead of an
    element-wise pass over two tensors).  The gradient of ``res`` is the output gradient itself."""
    pending = getattr(w, "_ft_gather", None)
    if pending is not None:
        pending.complete_without_product()
    return torch_ops().linear(x, w, None, res, None)


def linear_bias(x, w, b, res=None):
    """``x w^T + b`` (``+ res``) with the additions in the GEMM epilogue, rounded once; the bias
    gradient (column sums) is summed by the weight gradient's product where its tiles leave room, else by a
    pass over the output gradient."""
    if getattr(w, "_ft_gather", None) is not None:
        y = bias_add(linear(x, w), b)
        return y if res is None else res + y
    return torch_ops().linear(x, w, b, res, None)


# ------------------------------------------------------------------ RMSNorm
class _RMSNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, eps):
        h = x.shape[-1]
        x2 = x.reshape(-1, h).contiguous()
        rows = x2.shape[0]
        y = torch.empty_like(x2)
        inv = torch.empty(rows, dtype=torch.float32, device=x.device)
        _check(cuda_lib().ft_rmsnorm_fwd(ptr(x2), ptr(w), ptr(y), ptr(inv), rows, h, float(eps),
                                         dtype_code(x.dtype), stream_handle()), "ft_rmsnorm_fwd")
        ctx.save_for_backward(x2, w, inv)
        return y.view(x.shape)

    @staticmethod
    def backward(ctx, dy):
        x2, w, inv = ctx.saved_tensors
        rows, h = x2.shape
        dy2 = dy.reshape(rows, h).contiguous()
        dx = torch.empty_like(x2)
        dw = torch.empty_like(w)
        lib = cuda_lib()
        part = torch.empty(lib.ft_rmsnorm_bwd_parts() * h, dtype=torch.float32, device=x2.device)
        _check(lib.ft_rmsnorm_bwd(ptr(x2), ptr(w), ptr(dy2), ptr(inv), ptr(dx), ptr(dw), ptr(part), rows,
                                  h, dtype_code(x2.dtype), stream_handle()), "ft_rmsnorm_bwd")
        return dx.view(dy.shape), dw, None


def rmsnorm(x, w, eps):
    return _RMSNorm.apply(x, w, eps)


def layernorm(x, w, b, eps):
    """LayerNorm through the register-resident row kernels (``ft_norm_fwd`` / ``ft_norm_bwd_into``)."""
    return torch_ops().norm(x, w, b, eps)


def rmsnorm_rows(x, w, eps):
    """RMSNorm through the same row kernels as ``layernorm`` (each row read once)."""
    return torch_ops().norm(x, w, None, eps)


def norm_residual(x, w, b, eps):
    """``(x, norm(x))``: LayerNorm with ``b``, RMSNorm without.  The backward adds the gradient that
    arrives at ``x`` to the gradient through the norm in the norm's kernel."""
    return torch_ops().residual_norm(x, w, b, eps)


_NORM_MAX_HIDDEN = None


def norm_rows_supported(hidden: int) -> bool:
    """Whether the row-resident norm kernels cover this hidden size (forward and backward)."""
    global _NORM_MAX_HIDDEN
    if _NORM_MAX_HIDDEN is None:
        lib = cuda_lib()
        _NORM_MAX_HIDDEN = min(lib.ft_norm_max_hidden(0), lib.ft_norm_max_hidden(1))
    return hidden % 8 == 0 and 0 < hidden <= _NORM_MAX_HIDDEN


def add_rmsnorm(x, r, w, eps):
    """``s = x + r`` and ``y = rmsnorm(s) * w`` in one kernel; the backward adds the gradient
    that arrives at ``s`` from its other consumer (the next residual add) to the gradient through
    the norm inside the norm's backward kernel, so neither direction has an add pass."""
    return torch_ops().add_norm(x, r, w, None, eps)


def add_layernorm(x, r, w, b, eps):
    """``s = x + r`` and ``layernorm(s)`` likewise."""
    return torch_ops().add_norm(x, r, w, b, eps)


def bias_add(x, bias):
    """``x + bias`` over the last dimension, in place where ``x`` is contiguous; the backward
    gives the bias gradient (column sums) in one pass."""
    return torch_ops().bias_act(x, bias, 0)


def bias_gelu(x, bias):
    """``gelu(x + bias)`` (tanh form); the backward gives dx and the bias gradient in one pass."""
    return torch_ops().bias_act(x, bias, 1)


# --------------------------------------------------------------------- RoPE
def rope_heads_inplace(x, cos, sin, heads, d):
    """In-place rotary embedding of the leading ``heads`` heads of ``x [B, S, W]``."""
    if x.stride(2) != 1 or x.stride(0) != x.shape[1] * x.stride(1):
        raise ValueError("rope_heads_inplace needs a [B, S, W] tensor with contiguous rows")
    return torch_ops().rope_heads(x, cos.float().contiguous(), sin.float().contiguous(), heads, d)


class _Rope(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, cos, sin):
        B, S, H, D = x.shape
        xc = x if (x.stride(3) == 1 and x.stride(2) == D and x.stride(0) == S * x.stride(1)) \
            else x.contiguous()
        y = torch.empty(B, S, H, D, dtype=x.dtype, device=x.device)
        _check(cuda_lib().ft_rope(ptr(xc), xc.stride(1), ptr(y), y.stride(1), ptr(cos), ptr(sin), B * S,
                                  H, D, S, 1.0, dtype_code(x.dtype), stream_handle()), "ft_rope")
        ctx.save_for_backward(cos, sin)
        return y

    @staticmethod
    def backward(ctx, dy):
        cos, sin = ctx.saved_tensors
        dy = dy.contiguous()
        B, S, H, D = dy.shape
        dx = torch.empty_like(dy)
        _check(cuda_lib().ft_rope(ptr(dy), dy.stride(1), ptr(dx), dx.stride(1), ptr(cos), ptr(sin), B * S,
                                  H, D, S, -1.0, dtype_code(dy.dtype), stream_handle()), "ft_rope")
        return dx, None, None


def rope(x, cos, sin):
    return _Rope.apply(x, cos.float().contiguous(), sin.float().contiguous())


# ------------------------------------------------------------------- SwiGLU
def swiglu(gate_up):
    return torch_ops().swiglu(gate_up)


def linear_swiglu(x, w_gate_up):
    """``swiglu(x @ w.T)`` for ``w = [w_gate ; w_up]`` with the activation in the GEMM's epilogue.
    The ``[rows, 2F]`` projection is materialised only when a backward pass will need it (it is
    stored from the epilogue's registers, never read back in the forward)."""
    return torch_ops().linear_swiglu(x, w_gate_up)


# ---------------------------------------------------------------- attention
def _attn_impl() -> str:
    return os.environ.get("FLEXTRAIN_ATTN", "native")


def causal_attention(q, k, v, scale=None):
    """``q [B,S,H,D]``, ``k``/``v`` ``[B,S,Hkv,D]`` (views with a common row
    stride are fine) -> ``[B,S,H,D]``."""
    from . import attention
    return attention.causal_attention(q, k, v, scale)


# ------------------------------------------------- head + cross-entropy
class _KeptBytes:
    """A share of what the losses of a device may hold until their backward; given back by it or,
    with a loss that is dropped, by the garbage collector."""

    _held, _lock = {}, threading.RLock()

    def __init__(self, device, nbytes):
        self.device, self.nbytes = device, nbytes

    @classmethod
    def take(cls, device, nbytes, limit):
        """None where the share would exceed ``limit``."""
        with cls._lock:
            if cls._held.get(device, 0) + nbytes > limit:
                return None
            cls._held[device] = cls._held.get(device, 0) + nbytes
        return cls(device, nbytes)

    def give_back(self):
        with self._lock:
            self._held[self.device] -= self.nbytes
            self.nbytes = 0

    __del__ = give_back


class _LinearCrossEntropy(torch.autograd.Function):
    """Mean token cross-entropy of ``hidden @ weight.T`` without ever holding the
    full logits: rows are processed in chunks; forward keeps the per-row
    log-sum-exp and the logits of the last chunk, backward recomputes the other chunks',
    turns each chunk's into gradients in place and feeds the two gradient GEMMs.

    The last chunk's logits are kept because backward would allocate a buffer of that size
    anyway and starts with them: one sequence of 4096 tokens needs three products instead of
    four.  Not above ``KEEP_BYTES`` for all losses of a device that wait for their backward, so
    that a caller who sums many of them before one backward holds no more than that, and not
    where the last chunk fills only part of its buffer."""

    CHUNK = 4096
    KEEP_BYTES = 512 << 20

    @staticmethod
    def forward(ctx, hidden, weight, labels, ignore_index):
        lib = cuda_lib()
        n, h = hidden.shape
        v = weight.shape[0]
        hidden = hidden.contiguous()
        labels = labels.contiguous()
        dev = hidden.device
        lse = torch.empty(n, dtype=torch.float32, device=dev)
        loss_sum = torch.zeros(1, dtype=torch.float32, device=dev)
        count = torch.zeros(1, dtype=torch.int32, device=dev)
        _check(lib.ft_count_valid(ptr(labels), n, ignore_index, v, ptr(count), stream_handle()),
               "ft_count_valid")
        chunk = _LinearCrossEntropy.CHUNK
        logits = torch.empty(min(chunk, n), v, dtype=hidden.dtype, device=dev)
        for lo in range(0, n, chunk):
            rows = min(chunk, n - lo)
            gemm(hidden[lo:lo + rows], False, weight, False, rows, v, h, out=logits[:rows])
            _check(lib.ft_xent_fwd(ptr(logits), logits.stride(0), ptr(labels[lo:]), rows, v,
                                   ignore_index, ptr(lse[lo:]), ptr(loss_sum),
                                   dtype_code(logits.dtype), stream_handle()), "ft_xent_fwd")
        countf = count.float().clamp_(min=1.0)
        kept = None
        if n > 0 and n % min(chunk, n) == 0 and any(ctx.needs_input_grad[:2]):
            kept = _KeptBytes.take(dev, logits.nbytes, _LinearCrossEntropy.KEEP_BYTES)
        ctx.save_for_backward(hidden, weight, labels, lse, countf, logits if kept else None)
        ctx.kept = kept                              # until a backward has overwritten them
        ctx.ignore_index = ignore_index
        return (loss_sum / countf).squeeze(0)

    @staticmethod
    def backward(ctx, grad_out):
        hidden, weight, labels, lse, countf, logits = ctx.saved_tensors
        lib = cuda_lib()
        n, h = hidden.shape
        v = weight.shape[0]
        dev = hidden.device
        chunk = _LinearCrossEntropy.CHUNK
        scale = (grad_out.float().reshape(1) / countf).contiguous()
        dh = torch.empty_like(hidden)
        wg = weight.grad
        inplace = torch_ops().plain_backward() and wg is not None and wg.shape == weight.shape and wg.is_contiguous() \
            and wg.dtype == weight.dtype and wg.data_ptr() % 16 == 0
        dw = wg if inplace else torch.zeros_like(weight)
        kept, ctx.kept = ctx.kept, None
        have_last = kept is not None
        if not have_last:
            logits = torch.empty(min(chunk, n), v, dtype=hidden.dtype, device=dev)
        for lo in reversed(range(0, n, chunk)):
            rows = min(chunk, n - lo)
            hc = hidden[lo:lo + rows]
            lg = logits[:rows]
            if not (have_last and lo + rows == n):
                gemm(hc, False, weight, False, rows, v, h, out=lg)
            _check(lib.ft_xent_bwd(ptr(lg), lg.stride(0), ptr(labels[lo:]), rows, v, ctx.ignore_index,
                                   ptr(lse[lo:]), ptr(scale), 1.0, dtype_code(lg.dtype),
                                   stream_handle()), "ft_xent_bwd")
            gemm(lg, False, weight, True, rows, h, v, out=dh[lo:lo + rows])
            gemm(lg, True, hc, True, v, h, rows, out=dw, accumulate=True)
        if have_last:
            kept.give_back()
        return dh, (None if inplace else dw), None, None


def linear_cross_entropy(hidden, weight, labels, ignore_index=-100):
    return _LinearCrossEntropy.apply(hidden, weight, labels, int(ignore_index))
