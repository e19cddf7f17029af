"""LovaszSoftmaxV3 (CUDA, through the C ABI) against the CPU oracle and the golden files.
Inputs are continuous random logits, so error ties have measure zero."""
import os

import numpy as np
import pytest
import torch

from helpers import assert_grad_close, assert_loss_close, labels_with_ignores, run_module

pytestmark = pytest.mark.gpu


def _blocky_labels(gen, n, c, h, w, cell, ignore, frac):
    cells = torch.randint(0, c, (n, (h + cell - 1) // cell, (w + cell - 1) // cell), generator=gen)
    lb = cells.repeat_interleave(cell, 1).repeat_interleave(cell, 2)[:, :h, :w].contiguous()
    if frac > 0:
        lb[torch.rand(lb.shape, generator=gen) < frac] = ignore
    return lb


SHAPES = [(2, 5, 12, 11), (1, 19, 16, 16), (3, 4, 9, 7), (2, 7, 40, 52), (1, 3, 130, 127),
          (2, 19, 96, 96), (1, 2, 8, 8), (2, 40, 33, 20), (1, 300, 12, 12),
          # 512-pixel pipelined tiles: ragged second box, widest backward / forward class counts
          (2, 19, 26, 30), (1, 26, 24, 37), (1, 40, 30, 28),
          # odd pixel counts (no 16-byte aligned channel rows): a pixel's channels in one thread's registers
          # up to 40 classes (several 256-pixel groups per image), the tile kernel without TMA beyond
          (2, 19, 37, 41), (1, 33, 9, 31), (1, 41, 9, 31)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("per_image", [False, True])
@pytest.mark.parametrize("reduction", ["mean", "none"])
def test_matches_oracle(shape, per_image, reduction):
    import pytorch_loss as P
    from oracle import losses as O
    n, c, h, w = shape
    g = torch.Generator().manual_seed(sum(shape))
    logits = torch.randn(shape, generator=g)
    labels = labels_with_ignores(g, (n, h, w), c, 255, 0.1)
    want_loss, want_grad = O.lovasz_softmax(logits, labels, 255, reduction, per_image, dtype=torch.float64)
    loss, grad = run_module(P.LovaszSoftmaxV3(reduction, 255, per_image=per_image), logits.cuda(), labels.cuda())
    assert_loss_close(loss, want_loss.float(), atol=1e-6)
    assert_grad_close(grad, want_grad.float())
    ign = labels == 255
    assert bool((grad.cpu().transpose(0, 1)[:, ign] == 0).all())


def test_golden(golden_dir):
    import pytorch_loss as P
    z = np.load(os.path.join(golden_dir, "lovasz.npz"))
    for i in range(int(z["n_cases"])):
        ign = int(z[f"c{i}_hyper"][0])
        red = str(z[f"c{i}_reduction"])
        logits, labels = torch.from_numpy(z[f"c{i}_logits"]), torch.from_numpy(z[f"c{i}_labels"])
        loss, grad = run_module(P.LovaszSoftmaxV3(red, ign), logits.cuda(), labels.cuda())
        assert_loss_close(loss, torch.from_numpy(z[f"c{i}_loss_v1"]), atol=1e-6, what=f"c{i} loss")
        assert_grad_close(grad, torch.from_numpy(z[f"c{i}_grad_v1"]), what=f"c{i} grad")
        loss, grad = run_module(P.LovaszSoftmaxV3('none', ign, per_image=True), logits.cuda(), labels.cuda())
        assert_loss_close(loss, torch.from_numpy(z[f"c{i}_loss_per_image"]), atol=1e-6, what=f"c{i} per-image loss")
        assert_grad_close(grad, torch.from_numpy(z[f"c{i}_grad_per_image"]), what=f"c{i} per-image grad")


def test_multi_tile_segments_and_blocky_labels(monkeypatch):
    """Segments longer than one sort tile (8192 pixels), realistic label maps, absent classes; the
    pruned sort against the sort of every element."""
    import pytorch_loss as P
    from oracle import losses as O
    g = torch.Generator().manual_seed(77)
    logits = torch.randn(2, 19, 160, 200, generator=g)
    labels = _blocky_labels(g, 2, 17, 160, 200, 32, 255, 0.03)      # classes 17, 18 never occur
    for per_image in (False, True):
        want_loss, want_grad = O.lovasz_softmax(logits, labels, 255, 'none', per_image, dtype=torch.float64)
        crit = P.LovaszSoftmaxV3('none', 255, per_image=per_image)
        loss, grad = run_module(crit, logits.cuda(), labels.cuda())
        assert_loss_close(loss, want_loss.float(), atol=1e-6)
        assert_grad_close(grad, want_grad.float())
        monkeypatch.setenv("B200_LOVASZ_NO_PRUNE", "1")
        loss_full, grad_full = run_module(crit, logits.cuda(), labels.cuda())
        assert_loss_close(loss_full, loss, atol=1e-6)
        assert_grad_close(grad_full, grad, atol=1e-7)       # (a segment may take the 20-bit sort in one run only)
        # with every segment on the 30-bit sort the two runs rank identically: same bits
        monkeypatch.setenv("B200_LOVASZ_EXACT", "1")
        loss_full, grad_full = run_module(crit, logits.cuda(), labels.cuda())
        monkeypatch.delenv("B200_LOVASZ_NO_PRUNE")
        loss_pruned, grad_pruned = run_module(crit, logits.cuda(), labels.cuda())
        monkeypatch.delenv("B200_LOVASZ_EXACT")
        assert_loss_close(loss_full, loss_pruned, atol=1e-6)
        assert torch.equal(grad_full, grad_pruned)


def test_pruned_sort_cases(monkeypatch):
    """The sort drops elements past the last foreground element of their class (their dJ is exactly
    zero).  Cases that move that bound around: classes absent from some or all images, a saturated
    foreground pixel (error 0: nothing can be dropped), an image that is ignored entirely, and the
    unpruned path as a cross-check."""
    import pytorch_loss as P
    from oracle import losses as O
    g = torch.Generator().manual_seed(2024)
    n, c, h, w = 3, 7, 48, 44                                       # 2112 pixels per image: pipelined tiles
    base = torch.randn(n, c, h, w, generator=g)
    lab_few = torch.randint(0, 2, (n, h, w), generator=g)           # classes 2..6 absent everywhere
    lab_mixed = labels_with_ignores(g, (n, h, w), c, 255, 0.2)
    lab_mixed[1] = 255                                              # one image ignored entirely
    lab_mixed[2][lab_mixed[2] == 3] = 4                             # class 3 absent from image 2 only
    saturated = base.clone()
    saturated[0, :, 0, 0] = -40.0
    saturated[0, int(lab_mixed[0, 0, 0]) if lab_mixed[0, 0, 0] != 255 else 0, 0, 0] = 40.0
    lab_sat = lab_mixed.clone()
    if lab_sat[0, 0, 0] == 255:
        lab_sat[0, 0, 0] = 0
    cases = [(base, lab_few), (base * 6.0, lab_mixed), (saturated, lab_sat)]
    for logits, labels in cases:
        for per_image in (False, True):
            want_loss, want_grad = O.lovasz_softmax(logits, labels, 255, 'none', per_image, dtype=torch.float64)
            crit = P.LovaszSoftmaxV3('none', 255, per_image=per_image)
            loss, grad = run_module(crit, logits.cuda(), labels.cuda())
            assert_loss_close(loss, want_loss.float(), atol=1e-6)
            assert_grad_close(grad, want_grad.float())
            monkeypatch.setenv("B200_LOVASZ_NO_PRUNE", "1")
            monkeypatch.setenv("B200_LOVASZ_EXACT", "1")
            loss_full, grad_full = run_module(crit, logits.cuda(), labels.cuda())
            monkeypatch.delenv("B200_LOVASZ_NO_PRUNE")
            loss_pruned, grad_pruned = run_module(crit, logits.cuda(), labels.cuda())
            monkeypatch.delenv("B200_LOVASZ_EXACT")
            assert_loss_close(loss_full, loss, atol=1e-6)
            assert_grad_close(grad_full, grad, atol=1e-7)
            assert torch.equal(grad_full, grad_pruned)              # same ranks, same dJ, same gradient


def test_sorted_order_properties():
    """Size-independent checks on the raw C-ABI outputs: per segment the Jaccard gradients
    are non-negative and sum to 1 (J runs from 0 to 1) and the loss lies in [0, 1]."""
    from pytorch_loss import lovasz_softmax as L
    g = torch.Generator().manual_seed(78)
    logits = torch.randn(2, 6, 120, 150, generator=g).cuda()
    labels = labels_with_ignores(g, (2, 120, 150), 6, 255, 0.05).cuda()
    for per_image in (False, True):
        loss, jacc, _, _ = L.lovasz_forward(logits, labels, 255, per_image)
        seg = jacc.reshape(-1, jacc.shape[-1]).double()
        assert bool((seg >= 0).all())
        torch.testing.assert_close(seg.sum(1), torch.ones_like(seg[:, 0]), rtol=0, atol=1e-4)
        assert bool(((loss >= 0) & (loss <= 1)).all())


def test_all_ignored_and_reference_function_signature():
    import pytorch_loss as P
    logits = torch.randn(1, 4, 8, 8).cuda().requires_grad_(True)
    labels = torch.full((1, 8, 8), 255, dtype=torch.int64).cuda()
    loss = P.LovaszSoftmaxFunctionV3.apply(logits, labels, 255)
    assert loss.shape == (4,) and bool((loss == 0).all())
    loss.sum().backward()
    assert bool((logits.grad == 0).all())


def test_backward_twice_and_fp16_input():
    import pytorch_loss as P
    from oracle import losses as O
    g = torch.Generator().manual_seed(79)
    logits = torch.randn(2, 5, 20, 24, generator=g)
    labels = labels_with_ignores(g, (2, 20, 24), 5, 255, 0.1)
    x = logits.cuda().requires_grad_(True)
    loss = P.LovaszSoftmaxV3(ignore_index=255)(x, labels.cuda())
    g1, = torch.autograd.grad(loss, x, retain_graph=True)
    g2, = torch.autograd.grad(loss, x)
    assert torch.equal(g1, g2)                 # saved tensors are not clobbered
    want_loss, want_grad = O.lovasz_softmax(logits.half().float(), labels, 255, 'mean')
    loss16, grad16 = run_module(P.LovaszSoftmaxV3(ignore_index=255), logits.half().cuda(), labels.cuda())
    assert grad16.dtype == torch.float16
    assert_loss_close(loss16, want_loss, rtol=2e-3)
    assert_grad_close(grad16, want_grad, atol=2e-3 * float(want_grad.abs().max()), rtol=2e-3)


def test_unsupported_shapes_raise():
    import pytorch_loss as P
    with pytest.raises(RuntimeError):
        P.LovaszSoftmaxV3()(torch.randn(1, 1100, 4, 4).cuda(), torch.zeros(1, 4, 4, dtype=torch.int64).cuda())
    with pytest.raises(ValueError):
        P.LovaszSoftmaxV3(process_group=True)


# segments that are counted instead of sorted (from 262144 pixels and 4096 of a class on): pixel counts that are and
# are not a multiple of 4, pruned and not, saturated pixels (the shared last bin), a class below the limit, and one
# whose mistakes pile up in the first bin
@pytest.mark.parametrize("shape,per_image", [((1, 3, 512, 512), True), ((2, 5, 513, 515), True), ((3, 4, 301, 293), False)])
@pytest.mark.parametrize("kind", ["random", "trained", "saturated"])
def test_counted_segments_against_64_bits(shape, per_image, kind):
    import pytorch_loss as P
    from oracle import losses as O
    n, c, h, w = shape
    g = torch.Generator().manual_seed(h)
    x = torch.randn(shape, generator=g)
    y = torch.randint(0, c, (n, h // 16 + 1, w // 16 + 1), generator=g).repeat_interleave(16, 1).repeat_interleave(16, 2)
    y = y[:, :h, :w].contiguous()
    y[y == c - 1] = 0                                           # the last class: 64 pixels an image only
    y[:, :8, :8] = c - 1
    if kind != "random":
        lead = torch.rand((n, 1, h, w), generator=g) * (12 if kind == "trained" else 60) + 3
        other = torch.randint(0, c, (n, h, w), generator=g)
        wrong = torch.rand((n, h, w), generator=g) < 0.04
        x.scatter_add_(1, torch.where(wrong, other, y).unsqueeze(1), lead)
    y[torch.rand(y.shape, generator=g) < 0.03] = 255
    want, want_grad = O.lovasz_softmax(x, y, 255, "sum", per_image=per_image, dtype=torch.float64)
    leaf = x.cuda().requires_grad_(True)
    loss = P.LovaszSoftmaxV3("sum", 255, per_image=per_image)(leaf, y.cuda())
    grad, = torch.autograd.grad(loss, leaf)
    assert_loss_close(loss, want, rtol=2e-6)                    # sums of fp32 terms; the order inside a bin cancels
    # the 64-pixel class, sorted, sets both bounds (test_counted_classes_alone holds the counted ones to theirs): errors
    # that agree in their float32 rounding change places there, a step of dJ of at most 1/64^2
    assert float((grad.double().cpu() - want_grad).abs().max()) <= 1.0 / 64 ** 2
    # (swaps in the 64-pixel class, whose steps are the largest, alone make up 6e-5 of the norm in float32)
    assert float((grad.double().cpu() - want_grad).norm()) <= 2e-4 * float(want_grad.norm())
    again = P.LovaszSoftmaxV3("sum", 255, per_image=per_image)(leaf, y.cuda())
    assert torch.equal(torch.autograd.grad(again, leaf)[0], grad) and torch.equal(again, loss)


def test_more_segments_than_a_grid_has_rows():
    """4096 images x 17 classes = 69 632 segments per image: above 65 535, the limit of a grid's y and z."""
    import pytorch_loss as P
    n, c, h, w = 4096, 17, 4, 4
    g = torch.Generator().manual_seed(17)
    x, y = torch.randn((n, c, h, w), generator=g), torch.randint(0, c, (n, h, w), generator=g)
    leaf = x.double().requires_grad_(True)
    fg = torch.nn.functional.one_hot(y.reshape(n, -1), c).permute(0, 2, 1).double()          # [n, c, pixels]
    err, order = (fg - torch.softmax(leaf.reshape(n, c, -1), 1)).abs().sort(-1, descending=True)
    hit = fg.gather(-1, order)
    n_pos = fg.sum(-1, keepdim=True)
    jacc = 1.0 - (n_pos - hit.cumsum(-1)) / (n_pos + (1.0 - hit).cumsum(-1))
    want = (err * torch.diff(jacc, dim=-1, prepend=torch.zeros_like(n_pos))).sum(-1)
    want_grad, = torch.autograd.grad(want.sum(), leaf)
    xg = x.cuda().requires_grad_(True)
    loss = P.LovaszSoftmaxV3("none", 255, per_image=True)(xg, y.cuda())
    grad, = torch.autograd.grad(loss.sum(), xg)
    assert_loss_close(loss.reshape(n, c), want, rtol=1e-5, atol=1e-6)
    # two of the 16 pixels whose errors agree in float32 may change places, a step of at most 1/2 of a gradient term:
    # 17 M pairs of pixels agree to 6e-8 about once
    assert float((grad.double().cpu() - want_grad).norm()) <= 1e-3 * float(want_grad.norm())


def test_segment_with_few_elements_to_sort_keeps_all_key_bits(monkeypatch):
    """A large segment of which fewer than 32 768 elements count is ordered by all 30 key bits: the same dJ, bit for
    bit, as where every segment is (class 0 below: 6000 foreground pixels, about 16 000 elements with an error above
    their smallest one)."""
    import pytorch_loss as P
    g = torch.Generator().manual_seed(3)
    pixels = 512 * 512
    p0 = torch.full((pixels,), 1e-3)
    order = torch.randperm(pixels, generator=g)
    fg, mistakes = order[:6000], order[6000:16000]
    p0[fg] = 0.1 + 0.5 * torch.rand(6000, generator=g)
    p0[mistakes] = 0.4 + 0.5 * torch.rand(10000, generator=g)
    x = torch.stack([(p0 / (1 - p0)).log(), torch.zeros(pixels)]).reshape(1, 2, 512, 512).cuda()
    y = torch.ones(pixels, dtype=torch.int64)
    y[fg] = 0
    y = y.reshape(1, 512, 512).cuda()

    def gradient_of_class_0():
        leaf = x.clone().requires_grad_(True)
        loss = P.LovaszSoftmaxV3("none", 255)(leaf, y)
        return torch.autograd.grad(loss[0], leaf)[0], loss.detach()[0]

    grad, loss = gradient_of_class_0()
    monkeypatch.setenv("B200_LOVASZ_EXACT", "1")
    want, want_loss = gradient_of_class_0()
    assert int((want != 0).sum()) > 2 * 6000
    assert torch.equal(grad, want) and torch.equal(loss, want_loss)



@pytest.mark.parametrize("shape,per_image", [((1, 3, 512, 512), True), ((2, 5, 513, 515), True), ((3, 4, 301, 293), False)])
@pytest.mark.parametrize("kind", ["random", "trained"])
def test_counted_classes_alone(shape, per_image, kind):
    """Every class has tens of thousands of pixels and is counted.  The elements of a bin share a dJ: with b background
    elements in it that is off by about b / 2U of itself, U >= the class's pixels.  Random errors leave some tens of
    262 144 elements in each of 65 536 bins; confident mistakes share the bins next to 1, a few per cent of U, but
    their p (1 - p) is 1e-4 and less.  So a pixel is off by some 1e-4 of the largest gradient, and few are."""
    import pytorch_loss as P
    from oracle import losses as O
    n, c, h, w = shape
    g = torch.Generator().manual_seed(h + 1)
    x = torch.randn(shape, generator=g) * 1.4
    y = torch.randint(0, c, (n, h // 16 + 1, w // 16 + 1), generator=g).repeat_interleave(16, 1).repeat_interleave(16, 2)
    y = y[:, :h, :w].contiguous()
    if kind == "trained":
        other = torch.randint(0, c, (n, h, w), generator=g)
        wrong = torch.rand((n, h, w), generator=g) < 0.04
        x.scatter_add_(1, torch.where(wrong, other, y).unsqueeze(1), torch.rand((n, 1, h, w), generator=g) * 12 + 3)
    y[torch.rand(y.shape, generator=g) < 0.03] = 255
    want, want_grad = O.lovasz_softmax(x, y, 255, "sum", per_image=per_image, dtype=torch.float64)
    leaf = x.cuda().requires_grad_(True)
    loss = P.LovaszSoftmaxV3("sum", 255, per_image=per_image)(leaf, y.cuda())
    grad, = torch.autograd.grad(loss, leaf)
    assert_loss_close(loss, want, rtol=2e-6)
    assert float((grad.double().cpu() - want_grad).abs().max()) <= 1e-3 * float(want_grad.abs().max())
    assert float((grad.double().cpu() - want_grad).norm()) <= 5e-5 * float(want_grad.norm())


# equal logits: every element of a class falls into one bin (or two: foreground and background), whose counters a warp
# adds to together
@pytest.mark.parametrize("hw", [(512, 512), (513, 515)])
def test_counted_segments_of_equal_logits(hw):
    import pytorch_loss as P
    g = torch.Generator().manual_seed(hw[0])
    y = (torch.rand((1,) + hw, generator=g) < 0.3).long()
    y[torch.rand(y.shape, generator=g) < 0.03] = 255
    x = torch.zeros((1, 2) + hw).cuda().requires_grad_(True)
    loss = P.LovaszSoftmaxV3("sum", 255, per_image=True)(x, y.cuda())
    grad, = torch.autograd.grad(loss, x)
    assert_loss_close(loss, torch.tensor(1.0), rtol=2e-6)          # every error is 1/2 and a class's dJ add up to 1
    fg, bg = [], []                       # the mean dJ over all orders of foreground and background of each class
    for c in (0, 1):
        f, b = int((y == c).sum()), int((y == 1 - c).sum())
        mean = float((1.0 / torch.arange(f, f + b + 1, dtype=torch.float64)).mean())
        fg.append(mean)
        bg.append(f / (f * (f + b)) + f / b * (1.0 / (f + b) - mean))
    for c in (0, 1):
        d = torch.tensor([-fg[0], bg[1]] if c == 0 else [bg[0], -fg[1]], dtype=torch.float64)    # d loss / d p
        want = 0.5 * (d - 0.5 * d.sum())
        got = grad.detach().cpu().double().permute(0, 2, 3, 1)[y == c]
        # one float32 division each and a product
        assert float((got - want).abs().max()) <= 1e-6 * float(want.abs().max())
    assert not bool(grad.cpu().permute(0, 2, 3, 1)[y == 255].any())


@pytest.mark.parametrize("hw", [(512, 512), (513, 515)])
@pytest.mark.parametrize("kind", ["some", "saturated"])
def test_counted_segments_of_partly_equal_logits(hw, kind, monkeypatch):
    """Half of the pixels with equal logits, the others random or (the shared last bin) far apart: the loss of the
    sorted form, which does not depend on the order of equal errors, and bit for bit the same again."""
    import pytorch_loss as P
    g = torch.Generator().manual_seed(7)
    x = torch.randn((2, 5) + hw, generator=g) * (2 if kind == "some" else 40)
    x[:, :, ::2] = 0
    x[:, :, :40] = 0
    y = torch.randint(0, 5, (2,) + hw, generator=g)
    y[torch.rand(y.shape, generator=g) < 0.03] = 255
    leaf = x.cuda().requires_grad_(True)

    def step():
        loss = P.LovaszSoftmaxV3("none", 255, per_image=True)(leaf, y.cuda())
        return loss.detach(), torch.autograd.grad(loss.sum(), leaf)[0]

    loss, grad = step()
    again, grad_again = step()
    assert torch.equal(loss, again) and torch.equal(grad, grad_again)
    monkeypatch.setenv("B200_LOVASZ_EXACT", "1")
    want, _ = step()
    assert_loss_close(loss, want.cpu(), rtol=2e-6)


@pytest.mark.parametrize("mask", [float("-inf"), torch.finfo(torch.float32).min, float("nan")])
def test_counted_segments_with_masked_channels(mask, monkeypatch):
    """Channels masked at some pixels, or NaN there: the counted form agrees with the sorted one (all key bits), which
    the masks reach as errors of exactly 0 and 1; a NaN stays at its own pixels."""
    import pytorch_loss as P
    g = torch.Generator().manual_seed(11)
    x = torch.randn((1, 4, 520, 512), generator=g)
    y = torch.randint(0, 4, (1, 520, 512), generator=g)
    hit = torch.rand(y.shape, generator=g) < 0.02
    x[:, 3] = torch.where(hit, torch.tensor(mask), x[:, 3])
    leaf = x.cuda().requires_grad_(True)

    def step():
        loss = P.LovaszSoftmaxV3("none", 255, per_image=True)(leaf, y.cuda())
        return loss.detach().cpu(), torch.autograd.grad(loss.sum(), leaf)[0].cpu()

    loss, grad = step()
    monkeypatch.setenv("B200_LOVASZ_EXACT", "1")
    want, want_grad = step()
    assert_loss_close(loss, want, rtol=2e-6)
    assert torch.equal(torch.isnan(grad), torch.isnan(want_grad))
    if mask != mask:
        assert not bool(torch.isnan(grad.permute(0, 2, 3, 1)[~hit]).any())
    # (see test_counted_classes_alone: 65 000 pixels a class; the masked foreground pixels, errors of 1, share a bin)
    diff = torch.nan_to_num(grad - want_grad).double()
    assert float(diff.norm()) <= 1e-4 * float(torch.nan_to_num(want_grad).double().norm())
