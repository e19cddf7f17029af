"""Row layouts (M == 1): the lengths at which the row kernels change their walk, their lanes per row or
their register budget, with remainders, against the oracle in 64 bits."""
import pytest
import torch

from oracle import losses as O

pytestmark = pytest.mark.gpu

# classes: whole vectors / pairs / odd; 40 channels a lane at most, 256 and 2048 as bounds of the warp-by-row form
CLASSES = [2, 3, 4, 8, 19, 20, 32, 40, 41, 42, 80, 81, 150, 160, 162, 255, 256, 257, 513, 1000, 1023, 1024, 1028, 1280,
           1284, 1536, 1766, 2046, 2047, 2048]
# float32: sums of at most 2048 terms in a tree of packed adds and an approximate exponential of 2^-21;
# 16 bits: the result is rounded once (half 2^-11, bfloat16 2^-8 of the element)
TOL = {torch.float32: 3e-6, torch.float16: 1e-3, torch.bfloat16: 4e-3}


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kind", ["lsr", "lmargin"])
@pytest.mark.parametrize("rows", [1, 67, 2500])
def test_rows_against_64_bits(rows, kind, dtype):
    import pytorch_loss as P
    g = torch.Generator(device="cuda").manual_seed(rows)
    for c in CLASSES:
        x = (torch.randn(rows, c, generator=g, device="cuda") * 2).to(dtype)
        y = torch.randint(0, c, (rows,), generator=g, device="cuda")
        y[1::7] = -100
        up = torch.rand(rows, generator=g, device="cuda").to(dtype) + 0.5
        for reduction in ("none", "sum"):
            if kind == "lsr":
                crit = P.LabelSmoothSoftmaxCEV3(0.1, reduction, -100)
                want, want_grad = O.label_smooth_ce(x, y, 0.1, -100, reduction, torch.float64)
            else:
                crit = P.LargeMarginSoftmaxV3(0.3, reduction, -100)
                want, want_grad = O.large_margin_softmax(x, y, 0.3, -100, reduction, torch.float64)
            leaf = x.clone().requires_grad_(True)
            loss = crit(leaf, y)
            grad, = torch.autograd.grad(loss, leaf, up if reduction == "none" else None)
            with torch.no_grad():
                alone = crit(x, y)
            if reduction == "none":
                want_grad = want_grad * up.double().unsqueeze(1)
            tol_loss = TOL[dtype] if reduction == "none" else TOL[torch.float32]
            what = "%s c=%d %s %s" % (kind, c, dtype, reduction)
            assert float((loss.detach().double() - want).norm()) <= tol_loss * float(want.norm()) + 1e-6, what
            assert float((alone.double() - want).norm()) <= tol_loss * float(want.norm()) + 1e-6, what
            # (bfloat16 target and off-target parts are rounded once each, and their sum in the upstream product)
            assert float((grad.double() - want_grad).norm()) <= 2 * TOL[dtype] * float(want_grad.norm()) + 1e-6, what
            assert not bool(grad[y == -100].any()), what


@pytest.mark.parametrize("c", [64, 128, 252, 256])
def test_rows_with_labels_on_8_bytes(c):
    """Labels that do not start on 16 bytes (a slice) cannot be copied in bulk: the fused step is still there."""
    import pytorch_loss as P
    from pytorch_loss import _cabi
    g = torch.Generator(device="cuda").manual_seed(c)
    x = torch.randn(300, c, generator=g, device="cuda")
    y = torch.randint(0, c, (301,), generator=g, device="cuda")[1:]
    assert y.data_ptr() % 16 == 8
    assert _cabi.load_library().b200_softmax_fused_step_path(x.data_ptr(), y.data_ptr(), x.data_ptr(), 300, c, 1, _cabi.F32)
    want, want_grad = O.label_smooth_ce(x, y, 0.1, -100, "mean", torch.float64)
    leaf = x.clone().requires_grad_(True)
    loss = P.LabelSmoothSoftmaxCEV3(0.1, "mean", -100)(leaf, y)
    grad, = torch.autograd.grad(loss, leaf)
    assert abs(float(loss) - float(want)) <= 3e-6 * float(want)
    assert float((grad.double() - want_grad).norm()) <= 6e-6 * float(want_grad.norm())


# Many rows: several groups of rows in a stage and stages refilled many times, one to four lanes a row with the
# rotated walk, and (256 classes and more) warps that take several rows with the next one in flight.  Row counts are
# odd, so that the last stage is ragged.  Compared row by row: one row taken from another one's stage would show.
MANY = {300007: [2, 3, 19, 20, 21, 36, 40], 60001: [80, 150, 160, 162, 255], 20003: [256, 1000, 1024, 2047, 2048]}


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kind", ["lsr", "lmargin"])
@pytest.mark.parametrize("rows", MANY)
def test_many_rows_against_64_bits(rows, kind, dtype):
    import pytorch_loss as P
    g = torch.Generator(device="cuda").manual_seed(rows + 1)
    for c in MANY[rows]:
        x = (torch.randn(rows, c, generator=g, device="cuda") * 2).to(dtype)
        y = torch.randint(0, c, (rows,), generator=g, device="cuda")
        y[torch.rand(rows, generator=g, device="cuda") < 0.1] = -100
        up = torch.rand(rows, generator=g, device="cuda").to(dtype) + 0.5
        valid = y != -100
        oracle = (lambda: O.label_smooth_ce(x, y, 0.1, -100, "none", torch.float64)) if kind == "lsr" else \
            (lambda: O.large_margin_softmax(x, y, 0.3, -100, "none", torch.float64))
        want, want_grad = oracle()
        # (half: a gradient divided by the number of rows has too few bits)
        for reduction in ("none", "sum") if dtype is torch.float16 else ("none", "sum", "mean"):
            crit = P.LabelSmoothSoftmaxCEV3(0.1, reduction, -100) if kind == "lsr" else \
                P.LargeMarginSoftmaxV3(0.3, reduction, -100)
            leaf = x.clone().requires_grad_(True)
            loss = crit(leaf, y)
            grad, = torch.autograd.grad(loss, leaf, up if reduction == "none" else None)
            what = "%s c=%d %s %s" % (kind, c, dtype, reduction)
            if reduction == "none":
                scale = up.double().unsqueeze(1)
                assert float(((loss.detach().double() - want).abs() - TOL[dtype] * want.abs()).max()) <= 4e-6, what
            else:
                scale = 1.0 / float(valid.sum()) if reduction == "mean" else 1.0
                total = float(want.sum()) * scale
                assert abs(float(loss.detach()) - total) <= 3e-6 * abs(total), what
            ref = want_grad * scale
            # a row's gradient: rounded once in 16 bits, twice where the upstream gradient comes in
            err = (grad.double() - ref).norm(dim=1) - 2 * TOL[dtype] * ref.norm(dim=1)
            assert float(err.max()) <= (1e-6 if reduction != "mean" else 1e-6 * scale), what
            assert not bool(grad[~valid].any()), what


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("c", [3, 5, 19, 20, 41, 150, 255, 256, 1000, 2047, 2048])
def test_rows_with_channels_at_the_lowest_value(c, dtype):
    """Channels masked with the type's lowest value (the one that stands in for the target in large margin's sums
    among them): gradients as in 64 bits, and large margin's loss where its sum of differences is finite."""
    import pytorch_loss as P
    g = torch.Generator(device="cuda").manual_seed(c)
    rows = 64
    x = (torch.randn(rows, c, generator=g, device="cuda") * 2).to(dtype)
    y = torch.randint(0, c, (rows,), generator=g, device="cuda")
    low = torch.finfo(dtype).min
    off = ~torch.nn.functional.one_hot(y, c).bool()
    channel = torch.arange(c, device="cuda")[None, :]
    for what, masked in (("one", (channel == (torch.arange(rows, device="cuda") % 4)[:, None])),
                         ("several", (torch.rand(rows, c, generator=g, device="cuda") < 0.3) & (channel > 2)),
                         ("all but the target", torch.ones(rows, c, dtype=torch.bool, device="cuda"))):
        xm = x.masked_fill(masked & off, low)
        for kind in ("lmargin", "lsr"):
            if kind == "lmargin":
                crit, oracle = P.LargeMarginSoftmaxV3(0.3, "none", -100), O.large_margin_softmax(xm, y, 0.3, -100, "none", torch.float64)
            else:
                crit, oracle = P.LabelSmoothSoftmaxCEV3(0.1, "none", -100), O.label_smooth_ce(xm, y, 0.1, -100, "none", torch.float64)
            if kind == "lmargin" and what == "all but the target":
                # (the oracle's own differences of 1e38 cancel badly: q = 1 / (c - 1), p = 0 off the target)
                oracle = torch.zeros(rows, dtype=torch.float64, device="cuda"), torch.zeros_like(xm, dtype=torch.float64)
            leaf = xm.clone().requires_grad_(True)
            loss = crit(leaf, y)
            grad, = torch.autograd.grad(loss, leaf, torch.ones_like(loss))
            case = "%s c=%d %s, %s masked" % (kind, c, dtype, what)
            if kind == "lmargin" and what != "several":      # (label smooth sums the logits themselves)
                err = (loss.detach().double() - oracle[0]).abs() - TOL[dtype] * oracle[0].abs()
                assert float(err.max()) <= 4e-6, case
            assert float((grad.double() - oracle[1]).norm()) <= 2 * TOL[dtype] * float(oracle[1].norm()) + 1e-6, case
    if c % 2:    # a row of nothing but lowest values: every channel is as likely as the others
        leaf = torch.full((4, c), low, dtype=dtype, device="cuda").requires_grad_(True)
        up = torch.ones(4, dtype=dtype, device="cuda")
        grad, = torch.autograd.grad(P.LabelSmoothSoftmaxCEV3(0.1, "none", -100)(leaf, y[:4]), leaf, up)
        want = O.label_smooth_ce(torch.zeros(4, c, device="cuda"), y[:4], 0.1, -100, "none", torch.float64)[1]
        assert float((grad.double() - want).norm()) <= 2 * TOL[dtype] * float(want.norm())


def test_threads_that_need_different_amounts_of_shared_memory():
    """Two threads run one kernel at lengths whose stages take 131 and 82 KB: neither lowers the other's limit."""
    import threading

    import pytorch_loss as P
    failures = []

    def work(c):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                x = torch.randn(64, c, device="cuda").requires_grad_(True)
                y = torch.randint(0, c, (64,), device="cuda")
                crit = P.LabelSmoothSoftmaxCEV3(0.1, "sum", -100)
                for _ in range(300):
                    torch.autograd.grad(crit(x, y), x)
                torch.cuda.current_stream().synchronize()
        except Exception as exc:                              # noqa: BLE001  (reported by the main thread)
            failures.append((c, repr(exc)))

    threads = [threading.Thread(target=work, args=(c,)) for c in (2047, 1283)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
