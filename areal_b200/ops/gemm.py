"""bf16 GEMM on the tcgen05 kernel (``csrc/gemm_bf16.cu``) and the autograd
``linear`` built on it.

The three products of a linear layer run on one kernel by choosing operand
majors instead of materialising transposes:

* forward  ``y  = x W^T``  – both operands K-major
* dgrad    ``dx = dy W``   – ``W`` read MN-major
* wgrad    ``dW = dy^T x`` – both operands MN-major, fp32 output with optional
  accumulation into a main-grad buffer.

Counterpart of the cuBLAS-backed ``nn.Linear`` calls of the reference
(areal/experimental/models/archon/qwen3/model/model.py:103-293).
"""

from __future__ import annotations

import ctypes
import functools
from dataclasses import dataclass

import torch

from . import _lib, wgrad_defer


def _gemm_ref(a, b, a_mn, b_mn, bias, out_dtype, out, accumulate):
    A = a.t() if a_mn else a
    B = b.t() if b_mn else b
    c = A.float() @ B.float().t()
    if bias is not None:
        c = c + bias.float()
    if out is not None:
        if accumulate:
            out.add_(c.to(out.dtype))
        else:
            out.copy_(c.to(out.dtype))
        return out
    return c.to(out_dtype)


def _tma_operand(t: torch.Tensor) -> torch.Tensor:
    """``t`` with unit inner stride and a 16-byte aligned base and pitch, as TMA needs them. The extents stay what they are: a
    reduction rounded up beyond one operand's rows would read what lies behind it, and zeros times that need not be zero."""
    if t.stride(1) == 1 and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0:
        return t
    n = t.shape[1]
    if n % 8:
        return torch.nn.functional.pad(t, (0, -n % 8))[:, :n]
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def gemm(
    a: torch.Tensor,
    b: torch.Tensor,
    *,
    a_mn: bool = False,
    b_mn: bool = False,
    bias: torch.Tensor | None = None,
    out: torch.Tensor | None = None,
    out_dtype: torch.dtype = torch.bfloat16,
    accumulate: bool = False,
    bn: int = 0,
    chained: bool = False,
) -> torch.Tensor:
    """``C[M,N] = A B^T (+bias)``.

    ``a`` is ``[M,K]`` (``a_mn=False``) or ``[K,M]`` (``a_mn=True``); ``b`` is ``[N,K]``
    or ``[K,N]`` likewise. ``out`` may be a bf16 or fp32 2-D tensor with unit
    inner stride; ``accumulate`` adds to it. ``chained`` (skinny products): launched as programmatic dependents of the
    kernel before, which must not write ``b``; the weight is on its way while that kernel still runs.
    """
    if not _lib.use_cuda_kernels(a, b):
        return _gemm_ref(a, b, a_mn, b_mn, bias, out_dtype, out, accumulate)
    assert a.dtype == torch.bfloat16 and b.dtype == torch.bfloat16, "bf16 operands required"
    assert a.dim() == 2 and b.dim() == 2
    a, b = _tma_operand(a), _tma_operand(b)
    if a_mn:
        K, M = a.shape
    else:
        M, K = a.shape
    if b_mn:
        Kb, N = b.shape
    else:
        N, Kb = b.shape
    assert K == Kb, f"reduction dims differ: {K} vs {Kb}"
    if out is None:
        out = torch.empty((M, N), dtype=out_dtype, device=a.device)
        accumulate = False
    assert out.shape == (M, N) and out.stride(1) == 1
    assert out.dtype in (torch.bfloat16, torch.float32)
    ragged = (a.shape[1] % 8) or (b.shape[1] % 8)
    # skinny products (decode steps): too few output tiles for 148 SMs ⇒ split the K extent
    if (bn == 0 and not a_mn and not b_mn and not accumulate and out.dtype == torch.bfloat16 and out.stride(0) % 4 == 0
            and not ragged):
        splits = _splitk_plan(M, N, K)
        if splits:
            ws = torch.empty((splits * M, N), dtype=torch.float32, device=a.device)
            rc = _lib.kernels().b200_gemm_bf16_splitk(
                _lib.ptr(a), _lib.ptr(b), _lib.ptr(out), _lib.ptr(bias), _lib.ptr(ws), ctypes.c_int(M), ctypes.c_int(N),
                ctypes.c_int(K), ctypes.c_longlong(a.stride(0)), ctypes.c_longlong(b.stride(0)),
                ctypes.c_longlong(out.stride(0)), ctypes.c_int(splits), ctypes.c_int(int(chained)), _lib.stream_ptr())
            _lib.check(rc, "b200_gemm_bf16_splitk")
            _lib.count_launch(2)
            return out
    if bn == 0:
        bn = _tile_plan(M, N)
    rc = _lib.bind("b200_gemm_bf16", "pppp iii lll iiiii p")(
        a.data_ptr(), b.data_ptr(), out.data_ptr(), _lib.addr(bias), M, N, K, a.stride(0), b.stride(0), out.stride(0),
        a_mn, b_mn, out.dtype == torch.float32, accumulate, bn, _lib.stream_raw())
    _lib.check(rc, "b200_gemm_bf16")
    _lib.count_launch()
    return out


@functools.lru_cache(maxsize=4096)
def _tile_plan(M: int, N: int) -> int:
    """Tile of a product that is not split: 512 (256 x 256 on a pair of SMs), 256 or 128 (128 rows by so many columns on one).
    Whole rounds of tiles over the SMs, times what a tile takes. Forward / dgrad / wgrad of 16384 x 4096 x 2048 in TFLOP/s: 1495 / 1514 /
    1324 on pairs, 1318 / 1397 / 1251 with 256 columns, 1162 / 1239 / 1108 with 128; of 2600 x 2048 x 2048, where pairs leave
    40% of their second round empty, 734 / 757 / 589, 757 / 757 / 620 and 880 / 880 / 662."""
    # 512 is not chosen: a training step on pairs beside a rollout stream has stalled, and the cause is not proven
    cost = {256: 1.1 * -(-(-(-M // 128) * -(-N // 256)) // 148),
            128: 0.63 * -(-(-(-M // 128) * -(-N // 128)) // 148)}
    return min(cost, key=cost.get)


@functools.lru_cache(maxsize=4096)
def _splitk_plan(M: int, N: int, K: int) -> int:
    """Number of K slices of the skinny path for this shape (0: not a shape for it). The kernel walks items of 128 weight
    rows by a K slice, one CTA per SM, so a pass takes ``rounds of items * (reduction blocks of an item + its start)``, and each
    slice makes the reduction behind it longer. Up to 128 rows this is weighed in bytes against the partial sums that are
    written and read back (at half price: they stay in L2). One sequence of Qwen3-1.7B: 1.48 ms a step when slices cost nothing but
    their sums, 1.43 ms so. With more rows the sums of many slices cost more than they save (256 rows: 8.45 ms by that
    rule, 7.49 ms with slices for a single round of items), and a product with as many tiles as half the SMs is not split."""
    if M > 512 or N % 4 or K < 1024:
        return 0
    tiles, blocks = -(-M // 128) * -(-N // 128), -(-K // 64)
    if M > 128:
        splits = min(8, 148 // tiles, K // 256)
    else:
        rows = 32 if M <= 32 else 64 if M <= 64 else 128
        step = 148 * (128 + rows / 2) * 128  # bytes that all CTAs load per reduction block
        splits = min(range(1, min(16, blocks // 2) + 1),
                     key=lambda s: (-(-tiles * s // 148) * (-(-blocks // s) + 2) + 2 * s) * step + 4 * s * M * N)
    return splits if splits >= 2 else 0


def linear_pitched(x: torch.Tensor, w: torch.Tensor, bias: torch.Tensor | None = None) -> torch.Tensor:
    """``x @ w.T (+ bias)`` whose rows start 16-byte aligned whatever the number of columns: slices of them feed kernels
    that want aligned pitches."""
    N = w.shape[0]
    grad = torch.is_grad_enabled() and (x.requires_grad or w.requires_grad)
    if N % 8 == 0 or grad or not (_lib.use_cuda_kernels(x, w) and x.dtype == torch.bfloat16):
        return linear(x, w, bias)
    return gemm(x, w, bias=bias, out=torch.empty((x.shape[0], -(-N // 8) * 8), dtype=x.dtype, device=x.device)[:, :N])


@dataclass
class Slices:
    """A product whose reduction is still split: row ``r`` is the sum over ``s < n`` of the fp32 rows at ``s * stride + r *
    columns`` of ``ws``. The kernel that reads it does the sum."""

    ws: torch.Tensor
    stride: int
    n: int


def _tma_rows(*ts: torch.Tensor) -> bool:
    return all(t.stride(1) == 1 and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0 for t in ts)


def linear_slices(x: torch.Tensor, w: torch.Tensor) -> "torch.Tensor | Slices":
    """``x @ w.T``, as :class:`Slices` where the product is decode-sized and split over its reduction."""
    M, K = x.shape
    N = w.shape[0]
    splits = _splitk_plan(M, N, K) if x.dtype == torch.bfloat16 and _lib.use_cuda_kernels(x, w) else 0
    if not (splits and K % 8 == 0 and _tma_rows(x, w)):
        return linear(x, w)
    ws = torch.empty((splits * M, N), dtype=torch.float32, device=x.device)
    S, stride = ctypes.c_int(0), ctypes.c_longlong(0)
    rc = _lib.kernels().b200_gemm_bf16_splitk_partials(
        _lib.ptr(x), _lib.ptr(w), _lib.ptr(ws), ctypes.c_int(M), ctypes.c_int(N), ctypes.c_int(K),
        ctypes.c_longlong(x.stride(0)), ctypes.c_longlong(w.stride(0)), ctypes.c_int(splits), ctypes.byref(S),
        ctypes.byref(stride), _lib.stream_ptr())
    _lib.check(rc, "b200_gemm_bf16_splitk_partials")
    _lib.count_launch()
    return Slices(ws, stride.value, S.value)


def linear_relu2(x: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
    """``relu(x @ w.T)^2``. On the bf16 kernels the activation runs on the product's fp32 accumulators (for decode-sized
    products in the split-K reduction)."""
    grad = torch.is_grad_enabled() and (x.requires_grad or w.requires_grad)
    if not (_lib.use_cuda_kernels(x, w) and x.dtype in (torch.bfloat16, torch.float32)) or grad:
        return torch.relu(linear(x, w)).square()
    M, K = x.shape
    N = w.shape[0]
    if not (x.dtype == torch.bfloat16 and N % 8 == 0 and K % 8 == 0 and x.stride(1) == 1 and w.is_contiguous()
            and x.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0):
        z = linear(x, w)
        rc = _lib.kernels().b200_relu2(_lib.ptr(z), ctypes.c_longlong(z.numel()), ctypes.c_int(int(z.dtype == torch.float32)),
                                       _lib.stream_ptr())
        _lib.check(rc, "b200_relu2")
        _lib.count_launch()
        return z
    splits = _splitk_plan(M, N, K)
    ws = torch.empty((splits * M, N), dtype=torch.float32, device=x.device) if splits else None
    y = torch.empty((M, N), dtype=x.dtype, device=x.device)
    rc = _lib.kernels().b200_gemm_bf16_relu2(
        _lib.ptr(x), _lib.ptr(w), _lib.ptr(y), _lib.ptr(ws), ctypes.c_int(M), ctypes.c_int(N), ctypes.c_int(K),
        ctypes.c_longlong(x.stride(0)), ctypes.c_longlong(w.stride(0)), ctypes.c_int(splits), _lib.stream_ptr())
    _lib.check(rc, "b200_gemm_bf16_relu2")
    _lib.count_launch(2 if splits else 1)
    return y


@torch.no_grad()
def linear_rmsnorm(x: torch.Tensor, w: torch.Tensor, norm_w: torch.Tensor, eps: float,
                   residual: torch.Tensor | None = None, chained: bool = False):
    """``h = x @ w.T (+ residual)``; returns ``(rmsnorm(h) * norm_w, h)``: a decoder block's projection,
    residual add and following norm. For skinny (decode-step) shapes the residual add and the norm
    run inside the split-K reduction kernel (two launches instead of three, bit-identical results);
    other shapes run the separate kernels. Inference only. ``chained`` as in :func:`gemm`."""
    from . import fused

    M, K = x.shape
    N = w.shape[0]
    splits = _splitk_plan(M, N, K) if (_lib.use_cuda_kernels(x, w) and x.dtype == torch.bfloat16) else 0
    ok = (splits and N % 8 == 0 and N <= 8192 and K % 8 == 0 and x.stride(1) == 1 and w.stride(1) == 1
          and x.stride(0) % 8 == 0 and w.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0
          and (residual is None or residual.is_contiguous()) and norm_w.is_contiguous())
    if not ok:
        a = linear(x, w)
        if residual is None:
            return fused.rmsnorm(a, norm_w, eps), a
        return fused.rmsnorm(a, norm_w, eps, residual=residual)
    ws = torch.empty((splits * M, N), dtype=torch.float32, device=x.device)
    y = torch.empty((M, N), dtype=x.dtype, device=x.device)
    res_out = torch.empty((M, N), dtype=x.dtype, device=x.device)
    rc = _lib.kernels().b200_gemm_bf16_splitk_rmsnorm(
        _lib.ptr(x), _lib.ptr(w), None, _lib.ptr(ws), ctypes.c_int(M), ctypes.c_int(N), ctypes.c_int(K),
        ctypes.c_longlong(x.stride(0)), ctypes.c_longlong(w.stride(0)), ctypes.c_int(splits), _lib.ptr(residual),
        _lib.ptr(norm_w), _lib.ptr(y), _lib.ptr(res_out), ctypes.c_float(eps), ctypes.c_int(int(chained)), _lib.stream_ptr())
    _lib.check(rc, "b200_gemm_bf16_splitk_rmsnorm")
    _lib.count_launch(2)
    return y, res_out


@torch.no_grad()
def linear_swiglu(x: torch.Tensor, w: torch.Tensor, chained: bool = False) -> torch.Tensor:
    """``swiglu(x @ w.T)`` of a fused gate / up projection; for decode-sized products SwiGLU runs in the split-K reduction
    (the halves are rounded to bf16 in between, as by the separate kernels). Inference only. ``chained`` as in :func:`gemm`."""
    from . import fused

    M, K = x.shape
    N = w.shape[0]
    splits = _splitk_plan(M, N, K) if x.dtype == torch.bfloat16 and _lib.use_cuda_kernels(x, w) else 0
    if not (splits and N % 16 == 0 and K % 8 == 0 and _tma_rows(x, w)):
        return fused.swiglu(linear(x, w))
    ws = torch.empty((splits * M, N), dtype=torch.float32, device=x.device)
    out = torch.empty((M, N // 2), dtype=x.dtype, device=x.device)
    rc = _lib.kernels().b200_gemm_bf16_splitk_swiglu(
        _lib.ptr(x), _lib.ptr(w), _lib.ptr(out), _lib.ptr(ws), ctypes.c_int(M), ctypes.c_int(N // 2), ctypes.c_int(K),
        ctypes.c_longlong(x.stride(0)), ctypes.c_longlong(w.stride(0)), ctypes.c_int(splits), ctypes.c_int(int(chained)),
        _lib.stream_ptr())
    _lib.check(rc, "b200_gemm_bf16_splitk_swiglu")
    _lib.count_launch(2)
    return out


class _Linear(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, bias):
        shape = x.shape
        x2 = x.reshape(-1, shape[-1])
        y = gemm(x2, w, bias=bias, out_dtype=x.dtype)
        ctx.save_for_backward(x2, w)
        ctx.has_bias = bias is not None
        ctx.in_shape = shape
        return y.reshape(*shape[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x2, w = ctx.saved_tensors
        dy2 = dy.reshape(-1, dy.shape[-1])
        if dy2.dtype != x2.dtype:
            dy2 = dy2.to(x2.dtype)
        dx = dw = db = None
        if ctx.needs_input_grad[0]:
            dx = gemm(dy2, w, b_mn=True, out_dtype=x2.dtype).reshape(ctx.in_shape)
        if ctx.needs_input_grad[1]:
            main = getattr(w, "main_grad", None)
            queue = wgrad_defer.active()
            if queue is not None and (main is not None or w.is_leaf):
                # zero-bubble pipeline schedules: the weight-gradient GEMM is parked and runs in a later W action
                if main is not None:
                    queue.push(lambda: gemm(dy2, x2, a_mn=True, b_mn=True, out=main, accumulate=True))
                else:
                    queue.push(lambda: wgrad_defer.accumulate(
                        w, gemm(dy2, x2, a_mn=True, b_mn=True, out_dtype=w.dtype)))
            elif main is not None:
                # fp32 main-grad accumulation across micro-batches, fused in the epilogue
                gemm(dy2, x2, a_mn=True, b_mn=True, out=main, accumulate=True)
                dw = None
            else:
                dw = gemm(dy2, x2, a_mn=True, b_mn=True, out_dtype=w.dtype)
        if ctx.has_bias and ctx.needs_input_grad[2]:
            db = dy2.float().sum(0).to(dy2.dtype)
        return dx, dw, db


def linear(x: torch.Tensor, w: torch.Tensor, bias: torch.Tensor | None = None) -> torch.Tensor:
    """``x @ w.T + bias`` with forward and both backward products on the tcgen05 kernel."""
    if x.is_cuda and x.dtype == torch.bfloat16:
        return _Linear.apply(x, w, bias)
    if wgrad_defer.armed() and torch.is_grad_enabled():
        return wgrad_defer.SplitLinear.apply(x, w, bias)
    return torch.nn.functional.linear(x, w, bias)
