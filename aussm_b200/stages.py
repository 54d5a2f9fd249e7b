"""The AUSSM block's stages around the scan operator, in the scan's own (batch, channel, time) layout.

The reference's ``SSMauBlock`` (ai-modules/wavesAI/model/aussm.py:849-902) works token-major, ``(b, l, d)``,
and transposes to ``(b, d, l)`` and back around its convolution and around the operator (four transposing
copies per call, :858-864 and :888-897), applies the convolution through ``nn.Conv1d`` with padding and a
slice, and builds the step size with separate bias-add and softplus passes (:878-880).  Here every stage
produces its result directly in ``(b, d, l)``:

* ``project_tokens`` / ``project_channels`` / ``project_back``: the block's linear layers as matrix products
  whose output (or input) is channel-major, so no transposing copy exists.  Large products run on the
  library's split GEMM (float32-accurate, tcgen05), small ones as one batched product;
* ``causal_conv_bias``: depthwise causal convolution + bias, one pass (``aussm_b200_conv_pre_fwd/_bwd``);
* ``softplus_bias``: ``softplus(pre + scale * bias)``, one pass, in place (``aussm_b200_softplus_bias_fwd/_bwd``).

All functions are differentiable.  CUDA float32 tensors only.
"""
from __future__ import annotations

import torch
from torch import Tensor

from . import _lib
from .ops import _PLAIN, _eager, _f32c, _ptr, _stream, _workspace
from .variants import _gemm

__all__ = ["causal_conv_bias", "softplus_bias", "project_tokens", "project_channels", "project_back", "rms_norm",
           "rms_norm_residual"]

# Below this many floating-point operations a product runs as a batched library product over views; the split GEMM spends two passes over each operand on its FP16 parts before the product starts.
MIN_FLOP = 2.0e10


# ---------------------------------------------------------------------------
# element-wise stages
# ---------------------------------------------------------------------------
class _CausalConvBias(torch.autograd.Function):
    @staticmethod
    def forward(ctx, xs, weight, bias):
        b, d, l = xs.shape
        k = weight.shape[-1]
        lib = _lib.load()
        u = torch.empty_like(xs)
        w2 = weight.reshape(d, k).contiguous()
        with torch.cuda.device(xs.device):
            rc = lib.aussm_b200_conv_pre_fwd(_ptr(xs), _ptr(w2), _ptr(bias), _ptr(u), b, d, l, k, _stream(xs))
        _lib.check(rc, "causal_conv_bias")
        ctx.save_for_backward(xs, w2)
        ctx.has_bias = bias is not None
        ctx.wshape = weight.shape
        return u

    @staticmethod
    def backward(ctx, du):
        xs, w2 = ctx.saved_tensors
        b, d, l = xs.shape
        k = w2.shape[1]
        lib = _lib.load()
        du = du.contiguous()
        dxs = torch.empty_like(xs)
        dw = torch.empty_like(w2)
        dbias = torch.empty(d, device=xs.device, dtype=torch.float32) if ctx.has_bias else None
        with torch.cuda.device(xs.device):
            ws = _workspace(lib.aussm_b200_conv_pre_bwd_workspace_bytes(b, d), xs.device)
            rc = lib.aussm_b200_conv_pre_bwd(_ptr(du), _ptr(xs), _ptr(w2), _ptr(dxs), _ptr(dw), _ptr(dbias), b, d, l, k,
                                             _ptr(ws), ws.numel(), _stream(xs))
        _lib.check(rc, "causal_conv_bias backward")
        return dxs, dw.view(ctx.wshape), dbias


def causal_conv_bias(xs: Tensor, weight: Tensor, bias: Tensor = None) -> Tensor:
    """``conv1d(xs, weight, bias, padding=k-1, groups=d)[..., :l]`` for ``xs`` (b, d, l) and ``weight``
    (d, 1, k), k <= 4: the block's causal depthwise convolution (aussm.py:858-864) in one pass."""
    b, d, l = xs.shape
    return _CausalConvBias.apply(_f32c("xs", xs, (b, d, l)), _f32c("conv weight", weight),
                                 None if bias is None else _f32c("conv bias", bias, (d,)))


class _SoftplusBias(torch.autograd.Function):
    @staticmethod
    def forward(ctx, pre, bias, scale):
        b, d, l = pre.shape
        lib = _lib.load()
        dt = torch.empty_like(pre)
        with torch.cuda.device(pre.device):
            rc = lib.aussm_b200_softplus_bias_fwd(_ptr(pre), _ptr(bias), float(scale), _ptr(dt), b, d, l, _stream(pre))
        _lib.check(rc, "softplus_bias")
        ctx.save_for_backward(dt)
        ctx.scale = float(scale)
        ctx.has_bias = bias is not None
        return dt

    @staticmethod
    def backward(ctx, ddt):
        (dt,) = ctx.saved_tensors
        b, d, l = dt.shape
        lib = _lib.load()
        ddt = ddt.contiguous()
        dpre = torch.empty_like(dt)
        dbias = torch.empty(d, device=dt.device, dtype=torch.float32) if ctx.has_bias else None
        with torch.cuda.device(dt.device):
            ws = _workspace(lib.aussm_b200_softplus_bias_bwd_workspace_bytes(b, d), dt.device)
            rc = lib.aussm_b200_softplus_bias_bwd(_ptr(ddt), _ptr(dt), ctx.scale, _ptr(dpre), _ptr(dbias), b, d, l,
                                                  _ptr(ws), ws.numel(), _stream(dt))
        _lib.check(rc, "softplus_bias backward")
        return dpre, dbias, None


def softplus_bias(pre: Tensor, bias: Tensor = None, scale: float = 1.0) -> Tensor:
    """``softplus(pre + scale * bias[None, :, None])`` for ``pre`` (b, d, l): the block's step size
    (aussm.py:878-880, where dt_proj's bias enters a second time) in one pass."""
    b, d, l = pre.shape
    return _SoftplusBias.apply(_f32c("pre", pre, (b, d, l)), None if bias is None else _f32c("bias", bias, (d,)), scale)


# ---------------------------------------------------------------------------
# RMS norm
# ---------------------------------------------------------------------------
MAX_NORM_CHANNELS = 1024


def _rms_norm_ops(x: Tensor, weight: Tensor, eps: float) -> Tensor:
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * weight


def _norm_kernel_takes(x: Tensor, weight: Tensor) -> bool:
    """The kernels serve whole rows of quads in eager mode; everything else (other types and devices, odd widths,
    function transforms, forward-mode differentiation, tracers and dispatch modes) takes the plain operations."""
    return (type(x) in _PLAIN and type(weight) in _PLAIN and _eager()
            and x.is_cuda and x.dtype == torch.float32 and weight.dtype == torch.float32 and weight.device == x.device
            and weight.dim() == 1 and x.dim() >= 1 and x.shape[-1] == weight.shape[0] and x.numel() > 0
            and x.shape[-1] % 4 == 0 and x.shape[-1] <= MAX_NORM_CHANNELS)


def _aligned(t: Tensor) -> Tensor:
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


class _RMSNorm(torch.autograd.Function):
    """(norm(x), x): the second output carries the residual branch, whose gradient joins in the same pass."""

    @staticmethod
    def forward(ctx, x, weight, eps):
        xc, w = _aligned(x), _aligned(weight)
        d = xc.shape[-1]
        rows = xc.numel() // d
        y = torch.empty_like(xc)
        rstd = torch.empty(rows, device=xc.device, dtype=torch.float32)
        with torch.cuda.device(xc.device):
            rc = _lib.load().aussm_b200_rms_norm_fwd(_ptr(xc), _ptr(w), eps, _ptr(y), _ptr(rstd), rows, d, _stream(xc))
        _lib.check(rc, "rms_norm")
        ctx.save_for_backward(x, weight, rstd)
        ctx.eps = eps
        ctx.set_materialize_grads(False)
        return y, x.view_as(x)

    @staticmethod
    def backward(ctx, g, extra):
        x, weight, rstd = ctx.saved_tensors
        if g is None:
            return extra, None, None
        if torch.is_grad_enabled() or not _eager():    # a graph of the gradient is wanted: differentiable operations
            r = torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + ctx.eps)
            gw = g * weight
            dx = r * gw - x * r.pow(3) * (gw * x).mean(-1, keepdim=True)
            dw = (g * x * r).reshape(-1, x.shape[-1]).sum(0)
            return dx if extra is None else dx + extra, dw, None
        lib = _lib.load()
        xc, w, gc = _aligned(x), _aligned(weight), _aligned(g)
        ec = None if extra is None else _aligned(extra)
        d = xc.shape[-1]
        rows = xc.numel() // d
        dx, dw = torch.empty_like(xc), torch.empty(d, device=xc.device, dtype=torch.float32)
        with torch.cuda.device(xc.device):
            ws = _workspace(lib.aussm_b200_rms_norm_bwd_workspace_bytes(rows, d), xc.device)
            rc = lib.aussm_b200_rms_norm_bwd(_ptr(gc), _ptr(ec), _ptr(xc), _ptr(w), _ptr(rstd), _ptr(dx), _ptr(dw), rows, d,
                                             _ptr(ws), ws.numel(), _stream(xc))
        _lib.check(rc, "rms_norm backward")
        return dx, dw, None


def rms_norm(x: Tensor, weight: Tensor, eps: float = 1e-5) -> Tensor:
    """``x * rsqrt(mean(x^2, -1) + eps) * weight`` (the reference's RMSNorm, aussm.py:905-916) in one pass."""
    if not _norm_kernel_takes(x, weight):
        return _rms_norm_ops(x, weight, eps)
    return _RMSNorm.apply(x, weight, float(eps))[0]


def rms_norm_residual(x: Tensor, weight: Tensor, eps: float = 1e-5):
    """``(rms_norm(x), x)``: the pair a residual block needs; adding the second to the mixer's output lets the two
    gradients of x meet in the norm's backward pass instead of in a pass of their own."""
    if not _norm_kernel_takes(x, weight):
        return _rms_norm_ops(x, weight, eps), x
    return _RMSNorm.apply(x, weight, float(eps))


# ---------------------------------------------------------------------------
# linear layers with channel-major results
# ---------------------------------------------------------------------------
def _big(flop: float, *dims: int) -> bool:
    return flop >= MIN_FLOP


# Products below MIN_FLOP: one batched product per direction, in the layout the next stage reads.  torch.matmul folds
# the batch of a shared weight into rows, which copies the channel-major side before or after the product (six to
# eight transposing copies of a layer's training pass) and sums the weight's gradient over all b l tokens in the few
# tiles of one output (117 us each at 46080 tokens of 128 channels).  Training pass of SSMTS, 64 x 720 steps of width 128:
# 10.1 -> 6.9 ms of device time together with the row plans of block_stages.cu.  The gradients are ordinary operations, so
# they can be differentiated again.
class _BatchedTokens(torch.autograd.Function):
    """out[b] (m, l) = W (m, k) x[b]^T"""

    @staticmethod
    def forward(ctx, W, x):
        ctx.save_for_backward(W, x)
        return torch.bmm(W.expand(x.shape[0], -1, -1), x.transpose(1, 2))

    @staticmethod
    def backward(ctx, g):
        W, x = ctx.saved_tensors
        dW = _token_product(g, x) if ctx.needs_input_grad[0] else None
        dx = torch.bmm(g.transpose(1, 2), W.expand(x.shape[0], -1, -1)) if ctx.needs_input_grad[1] else None
        return dW, dx


class _BatchedChannels(torch.autograd.Function):
    """out[b] (m, l) = W (m, k) u[b] (k, l)"""

    @staticmethod
    def forward(ctx, W, u):
        ctx.save_for_backward(W, u)
        return torch.bmm(W.expand(u.shape[0], -1, -1), u)

    @staticmethod
    def backward(ctx, g):
        W, u = ctx.saved_tensors
        dW = _token_product(g, u.transpose(1, 2)) if ctx.needs_input_grad[0] else None
        du = torch.bmm(W.t().expand(u.shape[0], -1, -1), g) if ctx.needs_input_grad[1] else None
        return dW, du


class _BatchedBack(torch.autograd.Function):
    """out[b] (l, m) = y[b]^T (l, k) W^T"""

    @staticmethod
    def forward(ctx, W, y):
        ctx.save_for_backward(W, y)
        return torch.bmm(y.transpose(1, 2), W.t().expand(y.shape[0], -1, -1))

    @staticmethod
    def backward(ctx, g):
        W, y = ctx.saved_tensors
        gt = g.transpose(1, 2)
        dW = _token_product(gt, y.transpose(1, 2)) if ctx.needs_input_grad[0] else None
        dy = torch.bmm(W.t().expand(y.shape[0], -1, -1), gt) if ctx.needs_input_grad[1] else None
        return dW, dy


def _token_product(g: Tensor, x: Tensor) -> Tensor:
    """``sum_b g[b] x[b]`` for g (b, m, l), x (b, l, k): few tiles and a long contraction, so a single sequence is cut
    into pieces that run as batch entries (views) and the partial products are added."""
    b, m, l = g.shape
    if b == 1:
        pieces = 1
        while pieces < 64 and l % (2 * pieces) == 0 and l // (2 * pieces) >= 256:
            pieces *= 2
        if pieces > 1:
            return torch.bmm(g[0].unflatten(1, (pieces, -1)).transpose(0, 1), x[0].unflatten(0, (pieces, -1))).sum(0)
    return torch.bmm(g, x).sum(0)


def _batched(W: Tensor, x: Tensor, l: int) -> bool:
    """Whether a small product runs batched: the weight's gradient then has a partial product per batch entry, which
    may take twice the memory of the layer's input and output at most.  Under autocast the product's type is not its
    operands', which the gradients above do not undo: torch.matmul."""
    m, k = W.shape
    return (x.is_cuda and x.dtype == W.dtype == torch.float32 and x.numel() > 0 and m * k <= 2 * l * (m + k)
            and not torch.is_autocast_enabled("cuda") and _eager())


def _weight_grad(A: Tensor, a_mn: int, B: Tensor, b_mn: int, m: int, k: int, l: int, b: int) -> Tensor:
    """``dW[m][k] = sum_b sum_t A_b(m, t) B_b(k, t)`` for batched operands whose contraction index is time.

    ``x_mn == 0``: operand stored (rows, l) per batch entry, ``x_mn == 1``: stored (l, rows).  The output has few
    tiles and a very long contraction, so the time axis is cut into slices that run as independent batch entries
    of the split GEMM (one partial product each, through the strided entry point: the slices are views), and the
    partial products are added afterwards."""
    tiles = ((m + 127) // 128) * ((k + 255) // 256)
    slices = 1
    while tiles * slices * 2 <= 296 and l % (2 * slices) == 0 and (l // (2 * slices)) % 8 == 0 and l // (2 * slices) >= 512:
        slices *= 2
    ls = l // slices
    lib = _lib.load()
    part = torch.empty(b, slices, m, k, device=A.device, dtype=torch.float32)
    a_rows, b_rows = (m, k)
    lda, ldb = (l if a_mn == 0 else a_rows), (l if b_mn == 0 else b_rows)
    a_step = ls if a_mn == 0 else ls * a_rows           # floats between consecutive time slices
    b_step = ls if b_mn == 0 else ls * b_rows
    with torch.cuda.device(A.device):
        ws = _workspace(lib.aussm_b200_gemm_split3_workspace_bytes(m, k, ls, slices, a_mn, 1, b_mn, 1), A.device)
        for i in range(b):
            rc = lib.aussm_b200_gemm_split3_strided(
                A[i].data_ptr(), a_mn, lda, a_step, B[i].data_ptr(), b_mn, ldb, b_step, part[i].data_ptr(), k, m * k, m, k,
                ls, slices, 0, 0, _ptr(ws), ws.numel(), _stream(A))
            _lib.check(rc, "weight gradient (split GEMM)")
    return part.sum((0, 1))


class _ProjectTokens(torch.autograd.Function):
    """out[b] (m, l) = W (m, k) x[b]^T  for token-major x (b, l, k)."""

    @staticmethod
    def forward(ctx, W, x):
        m, k = W.shape
        b, l, _ = x.shape
        out = torch.empty(b, m, l, device=x.device, dtype=torch.float32)
        # A = W: (rows m, K) K-major, shared; B = x[b]: (rows l, K) K-major, batched
        _gemm(W, 0, 0, x, 0, 1, out, m, l, k, b, 0)
        ctx.save_for_backward(W, x)
        return out

    @staticmethod
    def backward(ctx, g):
        W, x = ctx.saved_tensors
        m, k = W.shape
        b, l, _ = x.shape
        g = g.contiguous()
        dW = dx = None
        if ctx.needs_input_grad[0]:
            # dW (m, k) = sum_b g[b] (m, K = l: K-major) x[b] (K = l rows, k contiguous: MN-major)
            dW = _weight_grad(g, 0, x, 1, m, k, l, b)
        if ctx.needs_input_grad[1]:
            dx = torch.empty_like(x)
            # dx[b] (l, k) = g[b]^T (l, K = m) W (K = m, k): g[b] stored (K rows, l contiguous) and W stored
            # (K rows, k contiguous): both MN-major
            _gemm(g, 1, 1, W, 1, 0, dx, l, k, m, b, 0)
        return dW, dx


def project_tokens(W: Tensor, x: Tensor) -> Tensor:
    """``einsum('mk,blk->bml')``: a linear layer applied to token-major ``x`` (b, l, k) whose result is
    channel-major (b, m, l)."""
    m, k = W.shape
    b, l, _ = x.shape
    if _big(2.0 * b * l * m * k):
        return _ProjectTokens.apply(_f32c("W", W), _f32c("x", x, (b, l, k)))
    if _batched(W, x, l):
        return _BatchedTokens.apply(W, x)
    return torch.matmul(W, x.transpose(1, 2))


def project_channels(W: Tensor, u: Tensor) -> Tensor:
    """``einsum('mk,bkl->bml')`` for channel-major ``u`` (b, k, l): result (b, m, l)."""
    m, k = W.shape
    b, _, l = u.shape
    if _big(2.0 * b * l * m * k):
        from .variants import _Projection
        return _Projection.apply(_f32c("W", W), _f32c("u", u, (b, k, l)))
    if _batched(W, u, l):
        return _BatchedChannels.apply(W, u)
    return torch.matmul(W, u)


class _ProjectBack(torch.autograd.Function):
    """out[b] (l, m) = y[b]^T (l, k) W^T  for channel-major y (b, k, l), W (m, k)."""

    @staticmethod
    def forward(ctx, W, y):
        m, k = W.shape
        b, _, l = y.shape
        out = torch.empty(b, l, m, device=y.device, dtype=torch.float32)
        # A = y[b]: (K = k rows, l contiguous) MN-major, batched; B = W: (rows m, K) K-major, shared
        _gemm(y, 1, 1, W, 0, 0, out, l, m, k, b, 0)
        ctx.save_for_backward(W, y)
        return out

    @staticmethod
    def backward(ctx, g):
        W, y = ctx.saved_tensors
        m, k = W.shape
        b, _, l = y.shape
        g = g.contiguous()
        dW = dy = None
        if ctx.needs_input_grad[0]:
            # dW (m, k) = sum_b g[b]^T (m, K = l) y[b]^T (K = l, k): g[b] stored (K = l rows, m contiguous)
            # MN-major, y[b] stored (k rows, K = l contiguous) K-major
            dW = _weight_grad(g, 1, y, 0, m, k, l, b)
        if ctx.needs_input_grad[1]:
            dy = torch.empty_like(y)
            # dy[b] (k, l) = W^T (k, K = m) g[b]^T (K = m, l): W stored (K rows, k contiguous) MN-major, shared;
            # g[b] stored (l rows, K = m contiguous) K-major
            _gemm(W, 1, 0, g, 0, 1, dy, k, l, m, b, 0)
        return dW, dy


def project_back(W: Tensor, y: Tensor, bias: Tensor = None) -> Tensor:
    """``einsum('mk,bkl->blm')`` (+ bias): a linear layer applied to channel-major ``y`` (b, k, l) whose result
    is token-major (b, l, m)."""
    m, k = W.shape
    b, _, l = y.shape
    if _big(2.0 * b * l * m * k):
        out = _ProjectBack.apply(_f32c("W", W), _f32c("y", y, (b, k, l)))
    elif _batched(W, y, l):
        out = _BatchedBack.apply(W, y)
    else:
        out = torch.matmul(y.transpose(1, 2), W.t())
    return out if bias is None else out + bias
