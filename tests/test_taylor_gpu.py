"""Taylor softmax / log-Taylor softmax / Taylor cross entropy (CUDA, through the C ABI) against
the CPU oracle and the golden file made from the reference's V1 functions."""
import math
import os

import numpy as np
import pytest
import torch

from helpers import assert_grad_close, assert_loss_close, labels_with_ignores

pytestmark = pytest.mark.gpu

# (shape, dim): 16-byte path, scalar path (odd inner size), one warp per row (dim last), dim 0
CASES = [((2, 19, 16, 24), 1), ((3, 7, 5, 7), 1), ((6, 33), 1), ((64, 1000), -1), ((5, 4, 6), 0),
         ((2, 3, 4, 40), 2), ((2, 150, 12, 12), 1), ((1, 2, 1, 1), 1),
         # 33..320 channels: channel slices over the threads of a block (4 slices to 160, 8 beyond), ragged ends
         ((1, 33, 5, 9), 1), ((2, 33, 6, 12), 1), ((3, 40, 70), 1), ((2, 161, 4, 10), 1), ((1, 161, 10, 10), 1),
         ((1, 320, 8, 8), 1), ((1, 321, 8, 8), 1),
         # rows of 64..1024 floats stay in a warp's registers (2 or 8 vectors per lane); 1028 does not
         ((40, 64), 1), ((33, 256), -1), ((9, 260), 1), ((17, 1024), 1), ((5, 1028), 1)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[0])) + "_d%d" % c[1])
@pytest.mark.parametrize("order", [2, 4, 8])
@pytest.mark.parametrize("use_log", [False, True])
def test_matches_oracle(case, order, use_log):
    import pytorch_loss as P
    from oracle import taylor as OT
    shape, dim = case
    g = torch.Generator().manual_seed(sum(shape) + order)
    x = torch.randn(shape, generator=g) * 1.5
    up = torch.randn(shape, generator=g)
    want_out, want_grad = OT.taylor_softmax(x, dim, order, use_log, upstream=up, dtype=torch.float64)
    xc = x.cuda().requires_grad_(True)
    out = P.taylor_softmax_v3(xc, dim, order, use_log)
    out.backward(up.cuda())
    assert out.shape == x.shape
    assert torch.allclose(out.detach().cpu().double(), want_out, atol=1e-6, rtol=1e-5)
    assert torch.allclose(xc.grad.cpu().double(), want_grad, atol=1e-5, rtol=1e-4)


def test_golden_and_modules(golden_dir):
    import pytorch_loss as P
    import taylor_softmax_cpp
    z = np.load(os.path.join(golden_dir, "taylor.npz"))
    for i in range(int(z["n_cases"])):
        dim, order, use_log = (int(v) for v in z[f"c{i}_hyper"])
        x, up = torch.from_numpy(z[f"c{i}_x"]).cuda(), torch.from_numpy(z[f"c{i}_up"]).cuda()
        out = taylor_softmax_cpp.taylor_softmax_forward(x, dim, order, bool(use_log))
        grad = taylor_softmax_cpp.taylor_softmax_backward(up, x, dim, order, bool(use_log))
        assert torch.allclose(out.cpu(), torch.from_numpy(z[f"c{i}_out"]), atol=1e-6, rtol=1e-5), i
        assert torch.allclose(grad.cpu(), torch.from_numpy(z[f"c{i}_grad"]), atol=1e-5, rtol=1e-4), i
    for i in range(int(z["n_ce_cases"])):
        order, ign = (int(v) for v in z[f"ce{i}_hyper"])
        logits = torch.from_numpy(z[f"ce{i}_logits"]).cuda().requires_grad_(True)
        labels = torch.from_numpy(z[f"ce{i}_labels"]).cuda()
        crit = P.TaylorCrossEntropyLossV3(n=order, ignore_index=ign, reduction=str(z[f"ce{i}_reduction"]))
        loss = crit(logits, labels)
        loss.backward()
        assert torch.allclose(loss.detach().cpu(), torch.from_numpy(z[f"ce{i}_loss"]), atol=1e-6, rtol=1e-5), i
        assert torch.allclose(logits.grad.cpu(), torch.from_numpy(z[f"ce{i}_grad"]), atol=1e-6, rtol=1e-5), i
    mod = P.TaylorSoftmaxV3(dim=1, n=4)
    y = mod(torch.randn(2, 5, 3, 3).cuda())
    assert torch.allclose(y.sum(dim=1), torch.ones(2, 3, 3).cuda(), atol=1e-6)
    y = P.LogTaylorSoftmaxV3(dim=1, n=2)(torch.randn(2, 5, 3, 3).cuda())
    assert torch.allclose(y.exp().sum(dim=1), torch.ones(2, 3, 3).cuda(), atol=1e-5)


def test_fp16_autocast_noncontiguous_empty_and_errors():
    import pytorch_loss as P
    from oracle import taylor as OT
    g = torch.Generator().manual_seed(4)
    x = torch.randn(2, 9, 6, 8, generator=g)
    want, _ = OT.taylor_softmax(x.half().float(), 1, 4, False)
    got = P.taylor_softmax_v3(x.half().cuda(), 1, 4, False)
    assert got.dtype == torch.float16
    assert torch.allclose(got.float().cpu(), want, atol=2e-3, rtol=2e-3)
    with torch.autocast("cuda", dtype=torch.float16):
        got = P.taylor_softmax_v3(x.half().cuda(), 1, 4, True)
    assert got.dtype == torch.float32                      # inputs are cast to fp32 under autocast
    xt = x.cuda().transpose(1, 3)                          # non-contiguous input
    want, _ = OT.taylor_softmax(x.transpose(1, 3), 1, 2, True)
    assert torch.allclose(P.taylor_softmax_v3(xt, 1, 2, True).cpu(), want, atol=1e-6, rtol=1e-5)
    assert P.taylor_softmax_v3(torch.empty(0, 5, 3).cuda(), 1, 2).shape == (0, 5, 3)
    with pytest.raises(RuntimeError):
        P.taylor_softmax_v3(x, 1, 4)                       # CPU tensor: gpu only
    with pytest.raises(RuntimeError):
        P.TaylorSoftmaxFunc.apply(x.cuda(), 1, 18, False)  # order above the supported 16


# class counts around the register budgets of the training step (8, 20, 24, 32, 40, 64, none above), pixel
# counts that are even, odd and shorter than a warp
@pytest.mark.parametrize("c", [1, 2, 8, 9, 20, 21, 25, 32, 33, 41, 64, 65])
@pytest.mark.parametrize("shape", [(16, 18), (7, 9), (2,)])
@pytest.mark.parametrize("order", [2, 8])
def test_cross_entropy_step_against_64_bits(c, shape, order):
    import pytorch_loss as P
    g = torch.Generator().manual_seed(c * 100 + order)
    x = torch.randn(3, c, *shape, generator=g)
    y = torch.randint(0, c, (3,) + shape, generator=g)
    y[torch.rand(y.shape, generator=g) < 0.2] = -1
    y.view(-1)[0] = 0
    for reduction in ("mean", "sum"):
        ref = x.double().requires_grad_(True)
        f = sum(ref.pow(i) / math.factorial(i) for i in range(order + 1))
        want = torch.nn.functional.nll_loss((f / f.sum(1, keepdim=True)).log(), y, ignore_index=-1, reduction=reduction)
        (want * 0.5).backward()
        leaf = x.cuda().requires_grad_(True)
        loss = P.TaylorCrossEntropyLossV3(order, -1, reduction)(leaf, y.cuda())
        first, = torch.autograd.grad(loss, leaf, torch.tensor(0.5, device="cuda"), retain_graph=True)
        first = first.clone()
        again, = torch.autograd.grad(loss, leaf, torch.tensor(0.5, device="cuda"))
        assert_loss_close(loss, want.float(), atol=1e-6)
        assert_grad_close(first, ref.grad)
        assert_grad_close(again, ref.grad)


def _taylor_64(x, y, n, reduction):
    leaf = x.detach().double().contiguous().requires_grad_(True)
    f = sum(leaf.pow(i) / math.factorial(i) for i in range(n + 1))
    loss = torch.nn.functional.nll_loss((f / f.sum(1, keepdim=True)).log(), y, ignore_index=-1, reduction=reduction)
    return loss.detach(), torch.autograd.grad(loss, leaf)[0]


@pytest.mark.parametrize("form", ["channels_last", "slice", "expanded_labels", "offset", "half_autocast", "bfloat16_autocast"])
def test_cross_entropy_step_takes_every_layout(form):
    """Layouts, strides and types that the one-kernel step accepts, against 64 bits."""
    import pytorch_loss as P
    g = torch.Generator().manual_seed(23)
    x = torch.randn(3, 7, 10, 12, generator=g).cuda()
    y = torch.randint(-1, 7, (3, 10, 12), generator=g).cuda()
    if form == "channels_last":
        x = x.contiguous(memory_format=torch.channels_last)
    elif form == "slice":
        x, y = x[:, 1:6, ::2, 1:], (y.clamp(max=4))[:, ::2, 1:]
    elif form == "expanded_labels":
        y = y[:1].expand(3, 10, 12)
    elif form == "offset":                                    # 4-byte aligned: one position a thread
        x = torch.randn(3 * 7 * 120 + 1, generator=g).cuda()[1:].view(3, 7, 10, 12)
    elif form.endswith("autocast"):
        x = x.to(torch.float16 if form.startswith("half") else torch.bfloat16)
    want, want_grad = _taylor_64(x, y, 4, "mean")
    leaf = x.detach().requires_grad_(True)
    crit = P.TaylorCrossEntropyLossV3(4, -1, "mean")
    with torch.autocast("cuda", dtype=leaf.dtype if form.endswith("autocast") else torch.float16, enabled=form.endswith("autocast")):
        assert crit._fused(leaf, y)
        loss = crit(leaf, y)
    grad, = torch.autograd.grad(loss, leaf)
    assert loss.dtype == torch.float32 and grad.dtype == leaf.dtype and grad.shape == leaf.shape
    assert_loss_close(loss, want)
    if form.endswith("autocast"):                             # (the gradient is rounded to the logits' type)
        assert float((grad.double() - want_grad).norm()) <= 4e-3 * float(want_grad.norm()) + 1e-7
    else:
        assert_grad_close(grad, want_grad)


def test_cross_entropy_step_with_nothing_to_count():
    import pytorch_loss as P
    x = torch.randn(2, 5, 6, 6, generator=torch.Generator().manual_seed(1)).cuda().requires_grad_(True)
    y = torch.full((2, 6, 6), -1, dtype=torch.int64).cuda()
    for reduction in ("mean", "sum"):
        loss = P.TaylorCrossEntropyLossV3(2, -1, reduction)(x, y)
        grad, = torch.autograd.grad(loss, x)
        assert torch.isnan(loss.detach()) if reduction == "mean" else float(loss.detach()) == 0.0
        assert not bool(grad.any())


@pytest.mark.parametrize("listener", ["global_hook", "instance_hook", "replaced_forward"])
def test_cross_entropy_calls_an_activation_that_somebody_listens_to(listener):
    import pytorch_loss as P
    crit = P.TaylorCrossEntropyLossV3(2, -1, "mean")
    act, calls = crit.taylor_softmax, []
    handle = None
    if listener == "global_hook":
        handle = torch.nn.modules.module.register_module_forward_hook(lambda m, i, o: calls.append(m) if m is act else None)
    elif listener == "instance_hook":
        handle = act.register_forward_hook(lambda m, i, o: calls.append(m))
    else:
        original = act.forward
        act.forward = lambda x: (calls.append(act), original(x))[1]
    try:
        g = torch.Generator().manual_seed(2)
        x = torch.randn(2, 5, 6, 6, generator=g).cuda().requires_grad_(True)
        crit(x, torch.randint(0, 5, (2, 6, 6), generator=g).cuda()).backward()
    finally:
        if handle is not None:
            handle.remove()
    assert calls == [act]
