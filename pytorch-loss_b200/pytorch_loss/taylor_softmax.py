"""Taylor softmax, log-Taylor softmax and Taylor cross entropy on the B200 CUDA library.

Drop-in for the reference's V3 classes and functions (pytorch_loss/taylor_softmax.py:15-35,
:76-98, :122-144, :175-198; extension functions csrc/taylor_softmax.cu:391-421):
`TaylorSoftmaxFunc`, `taylor_softmax_v3`, `TaylorSoftmaxV3(dim=1, n=2)`,
`LogTaylorSoftmaxV3(dim=1, n=2)`, `TaylorCrossEntropyLossV3(n=2, ignore_index=-1,
reduction='mean')`.  `dim` may be any dimension (negative values count from the end).
"""
import math

import torch
import torch.nn as nn
import torch.nn.functional as F
import torch.amp as amp

from . import _cabi


def _view(feat, dim):
    """(N, C, M) of `feat` around `dim`, and `dim` normalised."""
    if feat.dim() == 0:
        raise RuntimeError("taylor softmax needs at least one dimension")
    d = dim + feat.dim() if dim < 0 else dim
    if not 0 <= d < feat.dim():
        raise RuntimeError("dim %d out of range for a %d-dimensional tensor" % (dim, feat.dim()))
    shape = feat.shape
    return math.prod(shape[:d]), shape[d], math.prod(shape[d + 1:]), d


def taylor_softmax_forward(feat, dim, n, use_log):
    """The extension function of the reference: activation tensor like `feat`."""
    dev = _cabi.require_cuda(feat)
    feat = feat.contiguous()
    nn_, c, m, _ = _view(feat, int(dim))
    out = torch.empty_like(feat)
    lib = _cabi.load_library()
    with _cabi.on_device(dev):
        _cabi.check(lib.b200_taylor_softmax_forward(
            _cabi.ptr(feat), _cabi.ptr(out), nn_, c, m, _cabi.dtype_code(feat), int(n), int(bool(use_log)),
            _cabi.stream_ptr(dev)))
    return out


def taylor_softmax_backward(grad, feat, dim, n, use_log):
    """Gradient with respect to `feat` for the upstream gradient `grad` (same shape)."""
    dev = _cabi.require_cuda(grad, feat)
    feat = feat.contiguous()
    grad = grad.to(feat.dtype).contiguous()
    nn_, c, m, _ = _view(feat, int(dim))
    out = torch.empty_like(feat)
    lib = _cabi.load_library()
    with _cabi.on_device(dev):
        _cabi.check(lib.b200_taylor_softmax_backward(
            _cabi.ptr(grad), _cabi.ptr(feat), _cabi.ptr(out), nn_, c, m, _cabi.dtype_code(feat), int(n),
            int(bool(use_log)), _cabi.stream_ptr(dev)))
    return out


class TaylorSoftmaxFunc(torch.autograd.Function):
    """Reference pytorch_loss/taylor_softmax.py:17-34."""

    @staticmethod
    @amp.custom_fwd(cast_inputs=torch.float32, device_type='cuda')
    def forward(ctx, feat, dim=1, n=2, use_log=False):
        ctx.vars = feat, dim, n, use_log
        return taylor_softmax_forward(feat, dim, n, use_log)

    @staticmethod
    @amp.custom_bwd(device_type='cuda')
    def backward(ctx, grad_output):
        feat, dim, n, use_log = ctx.vars
        return taylor_softmax_backward(grad_output, feat, dim, n, use_log), None, None, None


def taylor_softmax_v3(inten, dim=1, n=4, use_log=False):
    assert n % 2 == 0 and n > 0
    return TaylorSoftmaxFunc.apply(inten, dim, n, use_log)


class TaylorSoftmaxV3(nn.Module):

    def __init__(self, dim=1, n=2):
        super().__init__()
        assert n % 2 == 0 and n > 0
        self.dim = dim
        self.n = n

    def forward(self, x):
        return taylor_softmax_v3(x, self.dim, self.n, use_log=False)


class LogTaylorSoftmaxV3(nn.Module):

    def __init__(self, dim=1, n=2):
        super().__init__()
        assert n % 2 == 0
        self.dim = dim
        self.n = n

    def forward(self, x):
        return taylor_softmax_v3(x, self.dim, self.n, use_log=True)


def _ce_step(logits, labels, n, ignore_index, mean):
    """The 'mean' / 'sum' training step in one pass over the logits: (record, final gradient)."""
    nn_, c, m = _cabi.split_shape(logits, labels)
    logits, labels = logits.contiguous(), labels.contiguous()
    lib = _cabi.load_library()
    dev = logits.device
    grads = torch.empty_like(logits)
    rec = _cabi.new_record(dev)
    ws = _cabi.reduce_workspace(dev)
    denom, flags = None, 0
    st, lp, wp, wn = _cabi.stream_ptr(dev), _cabi.ptr(labels), _cabi.ptr(ws), ws.numel()
    with _cabi.on_device(dev):
        if mean:       # (directly in front of the step's launch: it starts under the count's tail)
            count = _cabi.new_record(dev)
            denom = count.data_ptr() + _cabi.RECORD_COUNT
            _cabi.check(lib.b200_count_valid(lp, labels.numel(), int(ignore_index), count.data_ptr(), wp, wn, st))
            flags = _cabi.STEP_AFTER_COUNT
        _cabi.check(lib.b200_taylor_ce_step(
            _cabi.ptr(logits), lp, _cabi.ptr(grads), _cabi.ptr(rec), wp, wn, denom, nn_, c, m, _cabi.F32,
            int(ignore_index), int(n), flags, st))
    return rec, grads


class _TaylorCEFunc(torch.autograd.Function):
    """nll_loss of the log-Taylor softmax as one kernel for loss and gradient; backward multiplies by
    the upstream gradient (a kernel that leaves at once when that is 1)."""

    @staticmethod
    @amp.custom_fwd(cast_inputs=torch.float32, device_type='cuda')
    def forward(ctx, logits, labels, n, ignore_index, mean):
        rec, ctx.grads = _ce_step(logits, labels, n, ignore_index, mean)
        ctx.vars = logits, labels, n, ignore_index, mean
        return rec[4] if mean else rec[5]

    @staticmethod                             # (nothing in here depends on autocast)
    def backward(ctx, grad_output):
        grads, ctx.grads = ctx.grads, None
        if grads is None:                     # a second trip through the graph: the first scaled them in place
            _, grads = _ce_step(*ctx.vars)
        g = _cabi.scalar_gradient(grad_output)
        with _cabi.on_device(grads.device):
            _cabi.check(_cabi.load_library().b200_rescale_gradient(
                _cabi.ptr(grads), _cabi.ptr(g), None, grads.numel(), _cabi.F32, _cabi.stream_ptr(grads.device)))
        return grads, None, None, None, None


class TaylorCrossEntropyLossV3(nn.Module):
    """nll_loss of the log-Taylor softmax over dim 1 (reference :175-198).  Images of up to 64 classes
    ('mean' / 'sum', float32 logits or autocast, a gradient to produce) run loss and gradient as one
    kernel; everything else goes through the activation and torch's nll_loss."""

    def __init__(self, n=2, ignore_index=-1, reduction='mean'):
        super().__init__()
        assert n % 2 == 0
        self.taylor_softmax = LogTaylorSoftmaxV3(dim=1, n=n)
        self.reduction = reduction
        self.ignore_index = ignore_index

    def _fused(self, logits, labels):
        """The one-kernel step takes this call: what b200_taylor_ce_step_path accepts, and nobody listens to the
        activation or stands in for it."""
        act = self.taylor_softmax
        return (self.reduction in ('mean', 'sum') and type(act) is LogTaylorSoftmaxV3 and act.dim == 1 and
                2 <= act.n <= 16 and act.n % 2 == 0 and
                not (act._forward_hooks or act._forward_pre_hooks or act._backward_hooks or act._backward_pre_hooks or
                     'forward' in act.__dict__ or nn.modules.module._has_any_global_hook()) and
                logits.is_cuda and logits.requires_grad and torch.is_grad_enabled() and
                (logits.dtype == torch.float32 or
                 (torch.is_autocast_enabled('cuda') and logits.dtype in (torch.float16, torch.bfloat16))) and
                3 <= logits.dim() and logits.size(1) <= 64 and
                logits.size(0) * logits.size(1) < logits.numel() and      # (more than one pixel an image, no empty tensor)
                logits.numel() // logits.size(0) < 2 ** 31 and
                labels.device == logits.device and labels.dtype == torch.int64 and
                labels.shape == logits.shape[:1] + logits.shape[2:])

    def forward(self, logits, labels):
        if self._fused(logits, labels):
            return _TaylorCEFunc.apply(logits, labels, self.taylor_softmax.n, self.ignore_index, self.reduction == 'mean')
        log_probs = self.taylor_softmax(logits)
        return F.nll_loss(log_probs, labels, reduction=self.reduction, ignore_index=self.ignore_index)
