"""Autograd-aware fused operators backed by the sm_100a kernels.

Each function here is what a rewritten stage graph calls in place of one or
several ATen nodes of the exported model (``graph/rewrite.py`` does the
rewriting).  Forward and backward both run hand-written kernels; nothing in
here calls a library GEMM or attention.

Weight gradients go straight into a parameter's fp32 ``main_grad`` buffer when
it has one (the wgrad GEMM accumulates in its epilogue), so gradient
accumulation over micro-batches needs no separate add and no 16-bit rounding.
Reference counterpart: the ATen kernels run by src/torch/TorchDriver.cpp:566 and
the per-parameter ``grad`` buffers of src/comp/ParamStorage.cpp:33-191.
"""
from __future__ import annotations

import torch

from . import _lib
from . import kernels as K
from ..utils.config import conf
from .gemm import gemm, splits


# ----------------------------------------------------------------------------- RNG
class _Rng:
    """Counter-based dropout randomness: (seed, running offset).

    A recomputed forward reproduces its masks by restoring ``offset`` to the value
    it had when the original forward started (see ``get_state`` / ``set_state``),
    which is what the reference achieves by stashing the CUDA RNG state
    (src/comp/GraphConnector.cpp:395-457)."""

    def __init__(self):
        self.seed = 0x5EED
        self.offset = 0

    def next(self):
        self.offset += 1
        return self.seed, self.offset

    def get_state(self):
        return self.seed, self.offset

    def set_state(self, st):
        self.seed, self.offset = st


rng = _Rng()


def manual_seed(seed: int) -> None:
    rng.seed = int(seed) & 0x7FFFFFFFFFFFFFFF
    rng.offset = 0


def _main_grad(p):
    return None if p is None else getattr(p, "main_grad", None)


# ----------------------------------------------------------------------------- gradient reports
# The fused operators write weight gradients straight into the flat fp32 buffers, so autograd never sees them
# and no AccumulateGrad hook fires.  Instead every operator reports, at the END of its backward (after its last
# kernel that reads the weights was enqueued), which parameters it has just produced gradients for; the
# gradient reducer uses the reports to launch a bucket's reduction while backward is still running
# (parallel/fused_reduce.py).  The reference reduces after the whole backward (src/comp/Backward.cpp:100-107).
_grad_listener = None


def set_grad_listener(fn) -> None:
    global _grad_listener
    _grad_listener = fn
    if fn is not None or _lib.host_loaded():
        _lib.host().set_listener(fn)


def notify_grads(*params) -> None:
    if _grad_listener is not None:
        _grad_listener([p for p in params if p is not None])


def _kernel_ok(x) -> bool:
    return x.is_cuda and x.dtype in (torch.bfloat16, torch.float16)


def _aligned(t) -> bool:
    return t.data_ptr() % 16 == 0 and t.shape[-1] % 8 == 0 and t.shape[-1] > 0


def _dense16(t):
    """``t`` contiguous and on a 16-byte boundary, for kernels that read whole vectors."""
    return t if t.is_contiguous() and t.data_ptr() % 16 == 0 else t.clone(memory_format=torch.contiguous_format)


def _bias_ok(bias, n, dtype) -> bool:
    """None, or ``n`` values of the type the kernels read beside the operands."""
    return bias is None or (bias.dtype == dtype and bias.numel() == n)


def _bgrad(dy2, bias, mg):
    if bias is None:
        return None
    if mg is not None:
        K.colsum(dy2, out=mg)
        return None
    return K.colsum(dy2).to(bias.dtype)


def _host():
    """The native operators; like any autograd function without a batching rule they refuse functorch transforms."""
    if torch._C._are_functorch_transforms_active():
        raise RuntimeError("the fused operators do not support functorch transforms (vmap, grad, jvp, ...)")
    return _lib.host()


# ----------------------------------------------------------------------------- linear
def linear(x, weight, bias=None, act=None):
    """``act(x @ weight.T + bias)`` with ``act`` in (None, "gelu")."""
    if not (_kernel_ok(x) and weight.dtype == x.dtype and _aligned(x) and _aligned(weight) and weight.dim() == 2 and
            _bias_ok(bias, weight.shape[0], x.dtype)):
        y = torch.nn.functional.linear(x, weight, bias)
        return torch.nn.functional.gelu(y) if act == "gelu" else y
    return _host().linear(x, weight, bias, act == "gelu", _main_grad(weight), _main_grad(bias), None)


def mlp(x, w1, b1, w2, b2):
    """y = gelu(x W1^T + b1) W2^T + b2; the GELU derivative rides in the epilogue of a backward GEMM."""
    dt = x.dtype
    if not (_kernel_ok(x) and _aligned(x) and _aligned(w1) and _aligned(w2) and w1.dtype == dt and w2.dtype == dt and
            _bias_ok(b1, w1.shape[0], dt) and _bias_ok(b2, w2.shape[0], dt)):
        return torch.nn.functional.linear(torch.nn.functional.gelu(torch.nn.functional.linear(x, w1, b1)), w2, b2)
    return _host().mlp(x, w1, b1, w2, b2, _main_grad(w1), _main_grad(b1), _main_grad(w2), _main_grad(b2))


# ----------------------------------------------------------------------------- layer norm
def dropout_add_layer_norm(x, residual, gamma, beta, p: float = 0.0, eps: float = 1e-5, training: bool = True):
    """``LayerNorm(dropout(x, p) + residual)`` over the last dimension; the result has x's type.  The kernels want
    operands of one type and a residual of x's shape; parameters of another type are applied in fp32."""
    p = p if training else 0.0
    H, dt = x.shape[-1], x.dtype
    if not (_kernel_ok(x) and K.ln_supported(H) and gamma is not None and beta is not None and
            gamma.dtype == dt and beta.dtype == dt and gamma.numel() == H and beta.numel() == H and
            (residual is None or (residual.dtype == dt and residual.shape == x.shape))):
        h = torch.nn.functional.dropout(x, p, True) if p > 0 else x
        if residual is not None:
            h = h + residual
        if any(t is not None and t.dtype != h.dtype for t in (gamma, beta)):
            gamma, beta = (None if t is None else t.float() for t in (gamma, beta))
            return torch.nn.functional.layer_norm(h.float(), (H,), gamma, beta, eps).to(dt)
        return torch.nn.functional.layer_norm(h, (H,), gamma, beta, eps)
    h = _host()
    seed, offset = rng.next() if p > 0.0 else (0, 0)
    return h.layer_norm(x, residual, gamma, beta, float(p), float(eps), seed, offset, _main_grad(gamma),
                        _main_grad(beta))


# ----------------------------------------------------------------------------- element-wise
class _Dropout(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, p):
        ctx.p = p
        ctx.seed, ctx.offset = rng.next()
        return K.dropout(_dense16(x), p, ctx.seed, ctx.offset)

    @staticmethod
    def backward(ctx, dy):
        return K.dropout(_dense16(dy), ctx.p, ctx.seed, ctx.offset), None


def dropout(x, p: float, training: bool = True):
    if not training or p <= 0.0:
        return x
    if not _kernel_ok(x) or x.numel() == 0:
        return torch.nn.functional.dropout(x, p, True)
    return _Dropout.apply(x, float(p))


class _Gelu(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        xc = _dense16(x)
        ctx.save_for_backward(xc)
        return K.gelu(xc)

    @staticmethod
    def backward(ctx, dy):
        (x,) = ctx.saved_tensors
        return K.gelu_bwd(x, _dense16(dy))


def gelu(x):
    if not _kernel_ok(x):
        return torch.nn.functional.gelu(x)
    return _Gelu.apply(x)


def embedding(weight, ids, padding_idx: int = -1):
    if not (_kernel_ok(weight) and weight.shape[1] % 8 == 0 and weight.is_contiguous() and ids.dtype == torch.int64 and
            ids.is_cuda):
        return torch.nn.functional.embedding(ids, weight, None if padding_idx < 0 else padding_idx)
    return _host().embedding(weight, ids, padding_idx, _main_grad(weight))


# ----------------------------------------------------------------------------- attention
class _Attention(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, key_bias, p, scale):
        # q, k, v: [B, S, H, D] views
        seed, offset = rng.next() if p > 0.0 else (0, 0)
        o, lse = K.attn_fwd(q, k, v, key_bias, scale, p, seed, offset)
        ctx.save_for_backward(q, k, v, o, lse, key_bias)
        ctx.p, ctx.seed, ctx.offset, ctx.scale = p, seed, offset, scale
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, o, lse, key_bias = ctx.saved_tensors
        B, S, H, D = q.shape
        # one [B, S, 3, H, D] buffer so the three gradients are views a fused QKV consumer can use as is
        dqkv = torch.empty(B, S, 3, H, D, dtype=q.dtype, device=q.device)
        dq, dk, dv = K.attn_bwd(q, k, v, o, lse, do, key_bias, ctx.scale, ctx.p, ctx.seed, ctx.offset,
                                dq=dqkv[:, :, 0], dk=dqkv[:, :, 1], dv=dqkv[:, :, 2])
        return dq, dk, dv, None, None, None


def _attn_operand_ok(t):
    return t.stride(-1) == 1 and t.data_ptr() % 16 == 0 and all(s % 8 == 0 for s in t.stride()[:-1])


def sdpa(q, k, v, attn_mask=None, dropout_p: float = 0.0, is_causal: bool = False, scale=None):
    """Drop-in for ``F.scaled_dot_product_attention`` on [B, H, S, D] operands.

    The fused kernel handles head dim 64, no causal mask, and an additive mask that
    only depends on (batch, key) -- shape [B, 1, 1, S].  Anything else falls back to
    the ATen implementation."""
    ok = (_kernel_ok(q) and q.dim() == 4 and q.shape[-1] == 64 and not is_causal and k.shape == q.shape
          and v.shape == q.shape and k.dtype == q.dtype and v.dtype == q.dtype)
    key_bias = None
    if ok and attn_mask is not None:
        B, H, S, D = q.shape
        if attn_mask.dtype != torch.bool and tuple(attn_mask.shape) == (B, 1, 1, S):
            key_bias = attn_mask.reshape(B, S).float().contiguous()
        else:
            ok = False
    if ok:
        qs, ks, vs = (t.transpose(1, 2) for t in (q, k, v))  # [B, S, H, D] views
        if not all(_attn_operand_ok(t) for t in (qs, ks, vs)):
            qs, ks, vs = (t.clone(memory_format=torch.contiguous_format) for t in (qs, ks, vs))
        sc = float(scale) if scale is not None else q.shape[-1] ** -0.5
        o = _Attention.apply(qs, ks, vs, key_bias, float(dropout_p), sc)
        return o.transpose(1, 2)
    return torch.nn.functional.scaled_dot_product_attention(q, k, v, attn_mask=attn_mask, dropout_p=dropout_p,
                                                            is_causal=is_causal, scale=scale)


# ----------------------------------------------------------------------------- loss
def cross_entropy(logits, labels, num_classes=None, ignore_index: int = -100, weight: float = 1.0):
    """Mean cross entropy over rows whose label is not ``ignore_index``.

    ``logits`` may have more columns than ``num_classes`` (vocabulary padding): the extra
    columns are ignored and get a zero gradient.  Returns an fp32 scalar."""
    ld = logits.shape[-1]
    V = int(num_classes) if num_classes is not None else ld
    l2 = logits.reshape(-1, ld)
    if not (_kernel_ok(l2) and l2.stride(1) == 1 and (l2.shape[0] <= 1 or l2.stride(0) >= ld) and 0 < V <= ld and
            labels.dtype == torch.int64 and labels.is_cuda and labels.numel() == l2.shape[0]):
        return torch.nn.functional.cross_entropy(l2[:, :V].float(), labels.reshape(-1), ignore_index=ignore_index) * weight
    # the logits are dead after the loss: backward writes the gradient over them
    return _host().cross_entropy(l2, labels.reshape(-1).contiguous(), V, ignore_index, float(weight))


# ----------------------------------------------------------------------------- fused QKV projection + attention
def qkv_attention(x, wq, bq, wk, bk, wv, bv, attn_mask=None, dropout_p: float = 0.0, is_causal: bool = False,
                  scale=None, num_heads: int = 1):
    """Self-attention block input side: the three projections of ``x`` [B, S, hid] and the attention itself.
    Returns [B, S, H * D].  Falls back to separate projections + ``sdpa`` when the fused kernels do not apply."""
    B, S, _ = x.shape
    Ho = wq.shape[0]
    D = Ho // num_heads
    same = wk.shape == wq.shape and wv.shape == wq.shape and (bq is None) == (bk is None) == (bv is None)
    ok = (_kernel_ok(x) and same and D == 64 and not is_causal and _aligned(x) and _aligned(wq)
          and wq.dtype == x.dtype and wk.dtype == x.dtype and wv.dtype == x.dtype
          and all(_bias_ok(b, Ho, x.dtype) for b in (bq, bk, bv)))
    key_bias = None
    if ok and attn_mask is not None:
        if attn_mask.dtype != torch.bool and tuple(attn_mask.shape) == (B, 1, 1, S):
            key_bias = attn_mask.reshape(B, S).float().contiguous()
        else:
            ok = False
    if ok:
        sc = float(scale) if scale is not None else D ** -0.5
        # ONE projection GEMM over the stacked weights; the attention kernels read q / k / v as strided views of its
        # [B, S, 3, H, D] output and write dq / dk / dv into one buffer that the single dgrad GEMM consumes
        h = _host()
        ws, bs = [wq, wk, wv], [bq, bk, bv]
        streamed = any(getattr(t, "_rannc_host", None) is not None or getattr(t, "_rannc_window", False) for t in ws)
        seed, offset = rng.next() if dropout_p > 0.0 else (0, 0)
        return h.qkv_attention(x, ws, bs, key_bias, float(dropout_p), sc, num_heads, seed, offset,
                               [_main_grad(t) for t in ws], [_main_grad(t) for t in bs], streamed)
    q = linear(x, wq, bq).view(B, S, num_heads, D).transpose(1, 2)
    k = linear(x, wk, bk).view(B, S, num_heads, D).transpose(1, 2)
    v = linear(x, wv, bv).view(B, S, num_heads, D).transpose(1, 2)
    o = sdpa(q, k, v, attn_mask, dropout_p, is_causal, scale)
    return o.transpose(1, 2).reshape(B, S, Ho)


# ----------------------------------------------------------------------------- convolution / batch norm
def _nhwc(x):
    """[N, H, W, C] contiguous view of a logically NCHW tensor on a 16-byte boundary (a copy only if it is not
    channels-last yet, or starts elsewhere)."""
    cl = x.contiguous(memory_format=torch.channels_last)
    return (cl if cl.data_ptr() % 16 == 0 else cl.clone()).permute(0, 2, 3, 1)


def _conv_weight(w):
    """[Co, kh * kw * Ci] with the taps outermost (the order ``im2col`` produces): a view for 1x1 and channels-last
    filters, otherwise a copy made for this use.  It is not kept: nothing tells when the filter's values change (an
    update through ``.data`` or by a kernel leaves no trace on the parameter), and every micro-batch in flight
    would hold one as large as the filter."""
    Co, Ci, kh, kw = w.shape
    taps_last = w.detach().permute(0, 2, 3, 1)
    if not taps_last.is_contiguous() and K.pack_taps_ok(w):
        return K.pack_taps(w.detach())
    return taps_last.reshape(Co, kh * kw * Ci)


class _Conv2d(torch.autograd.Function):
    """Convolution as a tcgen05 GEMM over channels-last activations: the picked pixels for strided 1x1 kernels
    (unstrided ones are linear layers, see ``conv2d``), the padded image or the ``im2col`` matrix otherwise; input
    gradient by the same kernel or through the adjoint gather, weight gradient as one GEMM."""

    @staticmethod
    def _operand(x4, k, s, pad):
        if k == 1 and pad == 0:
            return x4[:, ::s, ::s, :].contiguous().reshape(-1, x4.shape[-1])
        return K.im2col(x4, k, s, pad)

    @staticmethod
    def _implicit(k, stride, padding, Ci, Co, H=0, W=0) -> bool:
        """Stride-1 "same" convolutions with a filter larger than 1x1 can run as an implicit GEMM: the producer of
        the GEMM reads the zero-padded activation tap by tap (a row shift per tap), so neither the k*k-fold
        ``im2col`` matrix nor its adjoint is ever written.  The product is taken over a grid with ``pad`` zero rows and
        columns on one side (border positions are computed and dropped), so small feature maps pay more in extra
        arithmetic, and in tiles that few rows leave empty, than the gather costs in traffic.
        ``conv_implicit_max_overhead`` bounds (H + 2 pad)(W + 2 pad) / (H W), the border on both sides: 1.15 at 28 x 28
        (the kernel's own grid 1.07), 1.31 at 14 x 14 (1.15).  Forward and backward of 32 fp16 images on the device,
        implicit / gathered in us: 28 x 28 x 512 288 / 456, x 1024 1036 / 1356, x 2048 4702 / 5000; 14 x 14 x 512
        115 / 158, x 1024 343 / 385, x 2048 1351 / 1265; 7 x 7 x 1024 153 / 168.  The line lies at 14 because of the host,
        which takes 250 us for the one and 200 for the other, longer than the device for most of the smaller layers."""
        if not (k > 1 and k % 2 == 1 and stride == 1 and padding == (k - 1) // 2 and Ci % 64 == 0 and Co % 64 == 0
                and k * k <= 49 and bool(conf("conv_implicit_gemm"))):
            return False
        if H > 0 and W > 0:
            over = (H + 2 * padding) * (W + 2 * padding) / float(H * W)
            return over <= float(conf("conv_implicit_max_overhead"))
        return True

    @staticmethod
    def _padded(x4, pad):
        """[N * Hp * Wp, C] rows of the channels-last image with ``pad`` zero columns behind every row and ``pad``
        zero rows behind every image (Hp = H + pad, Wp = W + pad).  In the flattened rows those also lie in FRONT of
        the next row and image, so one border serves both sides: the product over the padded grid costs 7 % more
        than the outputs at 28 x 28 instead of the 15 % of a border all around."""
        if x4.is_cuda and x4.is_contiguous() and x4.data_ptr() % 16 == 0:
            xp = K.pad_nhwc(x4, pad)
        else:
            xp = torch.nn.functional.pad(x4, (0, 0, 0, pad, 0, pad))
        return xp.reshape(-1, x4.shape[-1])

    @staticmethod
    def _wgrad32(dy2, act, shifts=None):
        """fp32 dy^T act (with ``shifts``: one block of columns per filter tap).  The GEMM splits a long K over the GPU
        only when it accumulates: a product it would split is added to zeros, any other is stored.  The parts are added
        in the order they arrive; ``torch.use_deterministic_algorithms`` keeps the product in one piece."""
        cols = act.shape[1] * (len(shifts) if shifts is not None else 1)
        Co = dy2.shape[1]
        split = not torch.are_deterministic_algorithms_enabled() and splits(Co, cols, dy2.shape[0]) > 1
        dw2 = (torch.zeros if split else torch.empty)(Co, cols, dtype=torch.float32, device=dy2.device)
        more = {} if shifts is None else {"wgrad_shifts": shifts}
        return gemm(dy2, act, trans_a=True, trans_b=False, out=dw2, accumulate=split, **more)

    @staticmethod
    def _fold(dw2, w, w_mg, k):
        """The tap-major fp32 weight gradient into the fp32 gradient buffer, or as a gradient of w's own type."""
        Co, Ci = w.shape[:2]
        if w_mg is not None:
            if w_mg.dtype == torch.float32 and K.wgrad_fold_few_ok(w_mg):
                K.wgrad_fold_few(dw2, w_mg, k * k)
            elif w_mg.dtype == torch.float32 and K.wgrad_fold_ok(w_mg):
                K.wgrad_fold(dw2, w_mg, k * k)
            else:
                w_mg.add_(dw2.view(Co, k, k, Ci).permute(0, 3, 1, 2))
            return None
        dw = torch.empty(w.shape, dtype=w.dtype, device=w.device)
        if K.wgrad_fold_few_ok(dw) and dw.dtype != torch.float32:
            K.wgrad_fold_few(dw2, dw, k * k)
            return dw
        if K.wgrad_fold_ok(dw) and dw.dtype != torch.float32:
            K.wgrad_fold(dw2, dw, k * k)
            return dw
        return dw.copy_(dw2.view(Co, k, k, Ci).permute(0, 3, 1, 2))

    @staticmethod
    def _shifts(k, pad, Wp):
        return [(r - pad) * Wp + (s - pad) for r in range(k) for s in range(k)]

    @staticmethod
    def forward(ctx, x, w, bias, stride, padding):
        N, C, H, W = x.shape
        Co, _, k, _ = w.shape
        x4 = _nhwc(x)
        Ho, Wo = K.conv_out_size(H, k, stride, padding), K.conv_out_size(W, k, stride, padding)
        implicit = _Conv2d._implicit(k, stride, padding, C, Co, H, W)
        if implicit:
            Hp, Wp = H + padding, W + padding
            y2 = torch.empty(N * H * W, Co, dtype=x.dtype, device=x.device)
            gemm(_Conv2d._padded(x4, padding), _conv_weight(w), bias=bias, out=y2,
                 conv={"taps": k * k, "shifts": _Conv2d._shifts(k, padding, Wp)},
                 row_map=(Hp, Wp, H, W, 0))
        else:
            a = _Conv2d._operand(x4, k, stride, padding)
            y2 = gemm(a, _conv_weight(w), bias=bias)
        ctx.save_for_backward(x4, w)
        ctx.meta = (stride, padding, bias, _main_grad(w), _main_grad(bias) if bias is not None else None, implicit)
        return y2.view(N, Ho, Wo, Co).permute(0, 3, 1, 2)

    @staticmethod
    def backward(ctx, dy):
        x4, w = ctx.saved_tensors
        stride, padding, bias, w_mg, b_mg, implicit = ctx.meta
        N, H, W, C = x4.shape
        Co, Ci, k, _ = w.shape
        dy4 = _nhwc(dy)
        dy2 = dy4.reshape(-1, Co)
        if implicit:
            Hp, Wp = H + padding, W + padding
            shifts = _Conv2d._shifts(k, padding, Wp)
            dyp = _Conv2d._padded(dy4, padding)                 # zero where the padded grid has no output
            dx = None
            if ctx.needs_input_grad[0]:
                # dx[j] = sum_t dy[j - shift_t] W_t : the same kernel with the shifts negated and tap t's
                # [Co, Ci] block of the weight matrix as the [K, N] operand
                dx2 = torch.empty(N * H * W, C, dtype=dy2.dtype, device=dy2.device)
                gemm(dyp, _conv_weight(w), trans_b=False, out=dx2,
                     conv={"taps": k * k, "shifts": [-v for v in shifts], "b_tap_cols": Ci, "n": Ci},
                     row_map=(Hp, Wp, H, W, 0))
                dx = dx2.view(N, H, W, C).permute(0, 3, 1, 2)
            dw = None
            if ctx.needs_input_grad[1]:
                # dW_t = dy^T x[. + shift_t] for all taps in one GEMM over the padded rows: a block of output
                # columns reads the activation with its tap's row shift
                dw = _Conv2d._fold(_Conv2d._wgrad32(dyp, _Conv2d._padded(x4, padding), shifts), w, w_mg, k)
            db = _bgrad(dy2, bias, b_mg) if (bias is not None and ctx.needs_input_grad[2]) else None
            notify_grads(w if w_mg is not None else None, bias if b_mg is not None else None)
            return dx, dw, db, None, None
        dx = None
        if ctx.needs_input_grad[0]:
            da = gemm(dy2, _conv_weight(w), trans_b=False)
            if k == 1 and padding == 0:
                dx4 = torch.zeros(N, H, W, C, dtype=da.dtype, device=da.device)
                dx4[:, ::stride, ::stride, :] = da.view(N, -1, dx4[:, ::stride, ::stride, :].shape[2], C)
            else:
                dx4 = K.col2im(da, N, H, W, C, k, stride, padding)
            dx = dx4.permute(0, 3, 1, 2)
        dw = None
        if ctx.needs_input_grad[1]:
            a = _Conv2d._operand(x4, k, stride, padding)
            if k == 1 and w_mg is not None:
                gemm(dy2, a, trans_a=True, trans_b=False, out=w_mg.view(Co, Ci), accumulate=True)
            else:
                dw = _Conv2d._fold(_Conv2d._wgrad32(dy2, a), w, w_mg, k)
        db = _bgrad(dy2, bias, b_mg) if (bias is not None and ctx.needs_input_grad[2]) else None
        notify_grads(w if w_mg is not None else None, bias if b_mg is not None else None)
        return dx, dw, db, None, None


def _pair(v):
    if isinstance(v, (list, tuple)):
        return int(v[0]), int(v[1])
    return int(v), int(v)


def conv2d(x, weight, bias=None, stride=1, padding=0, dilation=1, groups=1):
    """``torch.nn.functional.conv2d`` for square kernels, groups = 1, dilation = 1 and channel counts that are
    multiples of 8 on the kernels; anything else goes to ATen."""
    s, p, d = _pair(stride), _pair(padding), _pair(dilation)
    Co, Ci, kh, kw = weight.shape
    ok = (_kernel_ok(x) and weight.dtype == x.dtype and groups == 1 and d == (1, 1) and kh == kw and s[0] == s[1] and
          p[0] == p[1] and Ci % 8 == 0 and Co % 8 == 0 and x.dim() == 4 and isinstance(p[0], int) and
          _bias_ok(bias, Co, x.dtype))
    if not ok:
        return torch.nn.functional.conv2d(x, weight, bias, stride, padding, dilation, groups)
    if kh == 1 and s[0] == 1 and p[0] == 0:
        # a 1x1 convolution is the linear layer over the pixels of the channels-last activation
        return _host().conv1x1(x, weight, bias, _main_grad(weight), _main_grad(bias))
    return _Conv2d.apply(x, weight, bias, s[0], p[0])


def batch_norm_act(x, gamma, beta, running_mean, running_var, training: bool = True, momentum: float = 0.1,
                   eps: float = 1e-5, relu: bool = False, residual=None):
    """``relu(batch_norm(x) + residual)`` with ``relu`` and ``residual`` optional.  Training mode with affine
    parameters on the kernels; evaluation mode (running statistics) and other cases on ATen."""
    ok = (_kernel_ok(x) and training and x.dim() == 4 and x.shape[1] % 8 == 0 and gamma is not None and
          beta is not None and (residual is None or (residual.shape == x.shape and residual.dtype == x.dtype)))
    if not ok:
        y = torch.nn.functional.batch_norm(x, running_mean, running_var, gamma, beta, training, momentum, eps)
        if residual is not None:
            y = y + residual
        return torch.relu(y) if relu else y
    return _host().batch_norm_act(x, residual, gamma, beta, running_mean, running_var, float(momentum), float(eps),
                                  bool(relu), _main_grad(gamma), _main_grad(beta))
