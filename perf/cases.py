"""What the performance of this library is measured on: training steps (loss and gradient of the logits)
through the public modules of `pytorch_loss`, over the sizes, types, layouts and options that training
programs hand over.

A case is a dict of plain values: `op` (which module), `n`, `c`, `h`, `w` (h = 0: classification rows
[n, c]), `dtype`, `layout` ("nchw" / "nhwc"), `reduction`, `weight` (the factor of this loss in a sum of
losses, i.e. the upstream gradient) and, for Lovasz, `per_image` and `trained` (logits of a network that
has learnt the labels, against logits at the start of training).
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pytorch-loss_b200"))
import pytorch_loss  # noqa: E402

IGNORE = 255                      # (above 255 classes: -100)
SMOOTH, LAM, ALPHA, GAMMA, THRESH = 0.1, 0.3, 0.25, 2, 0.7
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


def _case(op, n, c, h=0, w=0, **more):
    case = {"op": op, "n": n, "c": c, "h": h, "w": w, "dtype": "f32", "layout": "nchw", "reduction": "mean",
            "weight": 1.0, "per_image": False, "trained": False}
    case.update(more)
    return case


def listed():
    return [
        # fine-tuning a classifier with a small batch: latency and launches, no bandwidth to speak of
        _case("lsr", 256, 1000, name="lsr_rows_small"),
        # a large classification batch with bfloat16 logits
        _case("lsr", 32768, 1000, dtype="bf16", name="lsr_rows_bf16"),
        # next-token prediction: long bfloat16 rows over a padded vocabulary
        _case("lsr", 16384, 32768, dtype="bf16", name="lsr_vocab_bf16"),
        # semantic segmentation, 19 classes, crops with a power-of-two size
        _case("lsr", 16, 19, 512, 512, name="lsr_seg"),
        # dense binary targets (heat maps, edges): elementwise
        _case("focal", 16, 1, 1024, 1024, name="focal_dense"),
        # segmentation with many classes
        _case("lmargin", 8, 150, 512, 512, name="lmargin_seg150"),
        # a half-precision channels-last network, an odd crop size and per-pixel loss weights
        _case("lmargin", 4, 150, 473, 473, dtype="f16", layout="nhwc", reduction="none", name="lmargin_nhwc_odd"),
        # Lovasz over the whole batch (the default) late in training
        _case("lovasz", 4, 19, 512, 512, trained=True, name="lovasz_batch"),
        # Lovasz per image on large images early in training
        _case("lovasz", 8, 19, 1024, 1024, per_image=True, name="lovasz_images"),
        # hard-example mining on odd crops, as one of several weighted heads
        _case("ohem", 8, 19, 769, 769, weight=0.4, trained=True, name="ohem_odd"),
        # Taylor cross entropy in the place of softmax cross entropy
        _case("taylor", 16, 19, 512, 512, name="taylor_seg"),
        # long-tailed class frequencies
        _case("pc", 16, 19, 512, 512, name="pc_seg"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of these ranges: batches, class counts and image sizes over their logarithm, odd ones among them."""
    family = rng.choice(["rows", "rows", "vocab", "seg", "seg", "seg", "focal", "lovasz", "ohem", "taylor"])
    dtype = rng.choice(["f32", "f32", "f16", "bf16"])
    weight = rng.choice([1.0, 1.0, 0.4])
    # (a gradient divided by the number of pixels does not fit half precision: sums or per-pixel weights there)
    red = rng.choice(["sum", "none"]) if dtype == "f16" else rng.choice(["mean", "mean", "none"])
    if red == "none":
        weight = 1.0
    if family == "rows":
        c = rng.choice([10, 100, 1000, _log_int(rng, 8, 2048)])
        op = rng.choice(["lsr", "lsr", "lmargin"])
        return _case(op, _log_int(rng, 32, 65536), c, dtype=dtype, reduction=red, weight=weight)
    if family == "vocab":
        c = rng.choice([8192, 16384, 32768, 8 * _log_int(rng, 512, 4096)])
        return _case("lsr", _log_int(rng, 256, min(16384, (1 << 28) // c)), c, dtype=dtype, reduction=red,
                     weight=weight)
    # images: square power-of-two crops, crops of 1 mod 8, and whatever size
    side = rng.choice([128, 256, 512, 1024, 8 * rng.randint(16, 96) + 1, _log_int(rng, 96, 1024)])
    h = side
    w = rng.choice([side, side, 2 * side if side <= 512 else side, _log_int(rng, 96, 1024)])
    c = rng.choice([19, 2, 21, 150, _log_int(rng, 2, 150)])
    if family in ("lovasz", "ohem", "taylor"):
        c = rng.choice([19, 2, 21, _log_int(rng, 2, 64)])
    most = {"seg": 1 << 27, "focal": 1 << 25, "lovasz": 1 << 26, "ohem": 1 << 26, "taylor": 1 << 27}[family]
    n = _log_int(rng, 1, max(1, min(16, most // (c * h * w))))
    if family == "focal":
        c = rng.choice([1, 1, 4, c])
        n = max(1, min(n, most // (c * h * w)))
        return _case("focal", n, c, h, w, dtype=dtype, reduction="sum" if dtype == "f16" else "mean", weight=weight)
    if family == "lovasz":
        return _case("lovasz", n, c, h, w, per_image=rng.random() < 0.5, trained=rng.random() < 0.5, weight=weight)
    if family == "ohem":
        return _case("ohem", n, c, h, w, trained=True, weight=weight)
    if family == "taylor":
        return _case("taylor", n, c, h, w, weight=weight)
    op = rng.choice(["lsr", "lmargin", "pc"])
    layout = rng.choice(["nchw", "nchw", "nhwc"]) if op != "pc" else "nchw"
    return _case(op, n, c, h, w, dtype=dtype, layout=layout, reduction=red, weight=weight)


# ---- inputs

def _ignore(case):
    return IGNORE if case["c"] <= IGNORE else -100


def _spatial(case):
    return [case["h"], case["w"]] if case["h"] else []


def _labels(case, g):
    """Class maps made of 32 x 32 cells, as objects are (rows: one class each); 3 % of the pixels are ignored."""
    n, c, sp = case["n"], case["c"], _spatial(case)
    if not sp:
        lb = torch.randint(0, c, (n,), generator=g, device="cuda")
    else:
        cells = torch.randint(0, c, (n, -(-sp[0] // 32), -(-sp[1] // 32)), generator=g, device="cuda")
        lb = cells.repeat_interleave(32, 1).repeat_interleave(32, 2)[:, :sp[0], :sp[1]].contiguous()
    return lb, torch.rand([n] + sp, generator=g, device="cuda") < 0.03


def _proportions(c):
    w = torch.arange(1, c + 1, dtype=torch.float64).reciprocal()
    return w / w.sum()


def _inputs(case, seed):
    """(logits, labels, upstream gradient of the per-pixel losses or None)."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 11)
    n, c, sp = case["n"], case["c"], _spatial(case)
    x = torch.randn([n, c] + sp, generator=g, device="cuda").mul_(math.sqrt(2.0))
    if case["op"] == "focal":
        y = (torch.rand([n, c] + sp, generator=g, device="cuda") < 0.1).to(DTYPES[case["dtype"]])
        return x.to(DTYPES[case["dtype"]]), y, None
    lb, ignored = _labels(case, g)
    if case["trained"]:
        # the right class leads by 3 to 15 at most pixels, another class does at 4 % of them
        lead = torch.rand([n, 1] + sp, generator=g, device="cuda").mul_(12.0).add_(3.0)
        wrong = torch.rand([n] + sp, generator=g, device="cuda") < 0.04
        other = torch.randint(0, c, [n] + sp, generator=g, device="cuda")
        x.scatter_add_(1, torch.where(wrong, other, lb).unsqueeze(1), lead)
    lb = lb.masked_fill_(ignored, _ignore(case))
    x = x.to(DTYPES[case["dtype"]])
    if case["layout"] == "nhwc":
        x = x.contiguous(memory_format=torch.channels_last)
    up = None
    if case["reduction"] == "none":
        up = (torch.rand([n] + sp, generator=g, device="cuda") + 0.5).to(x.dtype)
    return x, lb, up


def _criterion(case):
    ig, red = _ignore(case), case["reduction"]
    if case["op"] == "lsr":
        return pytorch_loss.LabelSmoothSoftmaxCEV3(SMOOTH, red, ig)
    if case["op"] == "lmargin":
        return pytorch_loss.LargeMarginSoftmaxV3(LAM, red, ig)
    if case["op"] == "focal":
        return pytorch_loss.FocalLossV3(ALPHA, GAMMA, red)
    if case["op"] == "lovasz":
        return pytorch_loss.LovaszSoftmaxV3(red, ig, per_image=case["per_image"])
    if case["op"] == "ohem":
        return pytorch_loss.OhemCELoss(THRESH, None, ig)
    if case["op"] == "taylor":
        return pytorch_loss.TaylorCrossEntropyLossV3(2, ig, red)
    return pytorch_loss.PCSoftmaxCrossEntropyV2(_proportions(case["c"]).tolist(), red, ig)


def prepare(case, seed):
    x, y, up = _inputs(case, seed)
    if up is None and case["weight"] != 1.0:
        up = torch.tensor(case["weight"], device="cuda")          # (reduced losses are float32)
    return {"criterion": _criterion(case), "logits": x.requires_grad_(True), "labels": y, "upstream": up}


def run(state):
    loss = state["criterion"](state["logits"], state["labels"])
    grad, = torch.autograd.grad(loss, state["logits"], state["upstream"])
    return {"loss": loss.detach(), "grad": grad}


# ---- what a step cannot do without

def _sizes(case):
    pixels = case["n"] * max(1, case["h"]) * max(1, case["w"])
    return pixels * case["c"], pixels, 4 if case["dtype"] == "f32" else 2


def work(case):
    """Logits and labels read once, gradient (and per-pixel losses) written once; about a dozen operations
    for each logit (maximum, exponential, sums, gradient)."""
    e, p, s = _sizes(case)
    if case["op"] == "focal":
        return {"bytes": 3 * s * e, "flops": 20 * e}
    per_pixel = (2 * s * p) if case["reduction"] == "none" else 0
    return {"bytes": 2 * s * e + 8 * p + per_pixel, "flops": 12 * e}


def tolerance(case):
    """Measured against 64 bits over the listed cases and drawn ones, times about four.  In 16 bits the
    gradient is rounded once.  Lovasz: where the errors of two pixels agree to the last bits their ranks
    may change places, and a rank is a large step where a class has few pixels.  Hard-example mining: a
    pixel whose score equals the last one that is kept may fall on either side."""
    if case["op"] == "lovasz":
        return {"rel": 1.2e-3, "max": 0.9}
    if case["op"] == "ohem":
        return {"rel": 1e-3, "max": 0.9}
    if case["dtype"] == "bf16":
        return {"rel": 1e-2, "max": 5e-2}
    if case["dtype"] == "f16":
        return {"rel": 1e-3, "max": 1.6e-2}
    return {"rel": 1e-6, "max": 1e-5}


# ---- the same in 64 bits

def _pixels_last(x):
    """[n, c, *] -> [n, c, m]"""
    return x.reshape(x.shape[0], x.shape[1], -1)


def _one_hot(x, lb):
    return torch.zeros_like(x).scatter_(1, lb.unsqueeze(1), 1.0)


def _softmax_losses(case, x, lb, valid):
    """Per-pixel loss [n, m] and its gradient [n, c, m] (both zero at ignored pixels), float64."""
    c = x.shape[1]
    if case["op"] == "lsr" or case["op"] == "ohem":
        eps = SMOOTH if case["op"] == "lsr" else 0.0
        logp = torch.log_softmax(x, 1)
        y = _one_hot(x, lb).mul_(1.0 - eps - eps / c).add_(eps / c)
        loss = -(logp * y).sum(1)
        grad = logp.exp_().mul_((c - 1) * (eps / c) + 1.0 - eps).sub_(y)
    elif case["op"] == "lmargin":
        k = 1.0 / (c - 1.0)
        hot = _one_hot(x, lb).bool()
        off = x.masked_fill(hot, -math.inf)
        logq = torch.log_softmax(off, 1)
        q = logq.exp()
        logq.masked_fill_(hot, 0.0)
        loss = ((q - k) * logq).masked_fill_(hot, 0.0).sum(1) * (LAM / 2.0)
        logp = torch.log_softmax(x, 1)
        loss = loss - logp.gather(1, lb.unsqueeze(1)).squeeze(1)
        qx = (q * x).sum(1, keepdim=True)
        grad = (q * (x + 1.0 - qx) - k).mul_(LAM / 2.0).masked_fill_(hot, -1.0).add_(logp.exp_())
    elif case["op"] == "pc":
        w = _proportions(c).to(x.device).view(1, c, 1)
        z = x + w.log()
        loss = torch.logsumexp(z, 1) - x.gather(1, lb.unsqueeze(1)).squeeze(1)
        grad = torch.softmax(z, 1) - _one_hot(x, lb)
    else:                                                     # taylor, order 2
        f = 1.0 + x + 0.5 * x * x
        s = f.sum(1, keepdim=True)
        loss = s.squeeze(1).log() - f.gather(1, lb.unsqueeze(1)).squeeze(1).log()
        grad = (1.0 + x) * (1.0 / s - _one_hot(x, lb) / f)
    v = valid.to(x.dtype)
    return loss * v, grad.mul_(v.unsqueeze(1))


def _exact_pixels(case, x, labels, up):
    ig = _ignore(case)
    if case["op"] == "ohem":
        scores = []
        for xi, li in zip(x.split(1), labels.split(1)):
            p = torch.softmax(_pixels_last(xi).double(), 1)
            flat = li.reshape(1, -1)
            s = p.gather(1, flat.masked_fill(flat == ig, 0).unsqueeze(1)).squeeze(1)
            scores.append(s.masked_fill_(flat == ig, 1.0).reshape(-1))
        scores = torch.cat(scores)
        n_min = labels.numel() // 16
        if n_min < labels.numel():
            hard = torch.sort(scores, stable=True).indices[:n_min]
            keep = scores <= THRESH
            keep[hard] = True
            labels = labels.masked_fill(~keep.view(labels.shape), ig)
    denom = float((labels != ig).sum())
    step = max(1, min(x.shape[0], (1 << 26) // max(1, x[0].numel())))
    losses, grads = [], []
    for i in range(0, x.shape[0], step):
        xi, li = _pixels_last(x[i:i + step]).double(), labels[i:i + step].reshape(labels[i:i + step].shape[0], -1)
        if not case["h"]:
            li = li.reshape(-1, 1)
        valid = li != ig
        lo, gr = _softmax_losses(case, xi, li.masked_fill(~valid, 0), valid)
        if case["reduction"] == "none":
            gr.mul_(up[i:i + step].reshape(lo.shape).double().unsqueeze(1))
            losses.append(lo.reshape(labels[i:i + step].shape))
        else:
            gr.mul_(case["weight"] / (denom if case["reduction"] == "mean" else 1.0))
            losses.append(lo.sum())
        grads.append(gr.view(x[i:i + step].shape))
        del xi, lo, gr
    if case["reduction"] == "none":
        loss = torch.cat(losses)
    else:
        loss = torch.stack(losses).sum() / (denom if case["reduction"] == "mean" else 1.0)
    return {"loss": loss, "grad": torch.cat(grads)}


def _exact_focal(case, x, y):
    p = torch.sigmoid(x)
    logp, log1p = torch.nn.functional.logsigmoid(x), torch.nn.functional.logsigmoid(-x)
    ce = y * ALPHA * logp + (1.0 - y) * (1.0 - ALPHA) * log1p
    d = (y - p).abs()
    coeff = -d.pow(GAMMA)
    d_coeff = GAMMA * d.pow(GAMMA - 1) * torch.sign(y - p) * p * (1.0 - p)
    d_ce = y * ALPHA * (1.0 - p) - (1.0 - y) * (1.0 - ALPHA) * p
    loss, scale = ce * coeff, case["weight"]
    if case["reduction"] == "mean":
        return {"loss": loss.mean(), "grad": (d_coeff * ce + d_ce * coeff) * (scale / x.numel())}
    return {"loss": loss.sum(), "grad": (d_coeff * ce + d_ce * coeff) * scale}


def _exact_lovasz(case, x, labels):
    n, c = x.shape[:2]
    flat, lab = _pixels_last(x), labels.reshape(n, -1)
    groups = [[i] for i in range(n)] if case["per_image"] else [list(range(n))]
    total, grad = x.new_zeros((), dtype=torch.float64), torch.zeros(flat.shape, dtype=torch.float64, device=x.device)
    scale = 1.0 / (c * len(groups))
    for images in groups:
        lb = torch.cat([lab[i] for i in images])
        probs = torch.cat([torch.softmax(flat[i].double(), 0) for i in images], 1)
        valid = lb != _ignore(case)
        dp = torch.zeros_like(probs)
        for k in range(c):
            fg = (lb == k) & valid
            err = torch.where(valid, (fg.double() - probs[k]).abs(), -torch.ones_like(probs[k]))
            err, order = torch.sort(err, descending=True)
            hits, counted = fg[order].double(), valid[order].double()
            inter = hits.sum() - hits.cumsum(0)
            union = hits.sum() + (counted - hits).cumsum(0)
            jacc = 1.0 - inter / union
            jacc[1:] -= jacc[:-1].clone()
            jacc *= counted
            total += (err * jacc).sum() * scale
            dp[k][order] = jacc * torch.where(hits > 0, -1.0, 1.0) * (scale * case["weight"])
        g = probs * (dp - (dp * probs).sum(0, keepdim=True)) * valid
        grad[images] = g.view(c, len(images), -1).transpose(0, 1)
    return {"loss": total, "grad": grad.view(x.shape)}


def exact(case, seed):
    x, y, up = _inputs(case, seed)
    x = x.detach()
    if case["op"] == "focal":
        return _exact_focal(case, x.double(), y.double())
    if case["op"] == "lovasz":
        return _exact_lovasz(case, x, y)
    return _exact_pixels(case, x, y, up)
