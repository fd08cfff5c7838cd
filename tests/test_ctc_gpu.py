"""
Fused CTC kernels (log-softmax + alpha/beta + gradient on packed logits) against torch.nn.functional.ctc_loss in fp32.
"""

import math
import pytest
import torch

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("lens,tlens,V,dtype", [
    ([30, 22, 5], [7, 3, 2], 50, torch.float32),
    ([334, 200, 120, 60], [11, 7, 4, 2], 10001, torch.bfloat16),
    ([12, 9], [4, 9], 33, torch.float32),       # second sequence: 9 labels in 9 frames (feasible only without repeats)
    ([6, 3], [2, 5], 17, torch.float32),        # second sequence infeasible -> loss 0, zero grad
    ([40], [0], 20, torch.float32),             # empty target
])
def test_ctc_loss_packed(lens, tlens, V, dtype):
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import ctc, _lib

    torch.manual_seed(0)
    B = len(lens)
    pack = PackInfo(torch.tensor(lens, dtype=torch.int32), torch.device("cuda"))
    blank = V - 1
    S = max(max(tlens), 1)
    targets = torch.randint(0, V - 1, (B, S), device="cuda", dtype=torch.int32)
    if len(lens) == 2 and tlens[1] == 9:
        targets[1] = torch.arange(9, device="cuda", dtype=torch.int32)  # no repeats
    tl = torch.tensor(tlens, dtype=torch.int32)
    logits = (torch.randn(pack.n, V, device="cuda") * 2).to(dtype).requires_grad_(True)
    w = torch.rand(B, device="cuda") + 0.5
    n0 = _lib.launch_count()
    loss = ctc.ctc_loss_packed(logits, pack, targets, tl, blank_index=blank)
    assert _lib.launch_count() > n0, "native kernels did not run"
    (loss * w).sum().backward()
    l32 = logits.detach().float().requires_grad_(True)
    padded = pack.unpack(l32)
    lp = torch.log_softmax(padded, dim=-1).transpose(0, 1)
    ref = torch.nn.functional.ctc_loss(lp, targets.long(), pack.lens_host.long(), tl.long(), blank=blank, reduction="none", zero_infinity=True)
    (ref * w).sum().backward()
    tol = 5e-2 if dtype == torch.bfloat16 else 1e-3
    torch.testing.assert_close(loss, ref, atol=tol, rtol=1e-3)
    gtol = 2e-2 if dtype == torch.bfloat16 else 1e-4
    torch.testing.assert_close(logits.grad.float(), l32.grad, atol=gtol, rtol=1e-2)


def _ctc_float64(x, pack, targets, tl, blank, w):
    """loss and gradient of every sequence in 64 bits"""
    x = x.detach().double().requires_grad_(True)
    lp, res, lo = torch.log_softmax(x, dim=-1), [], 0
    for b, (n, s) in enumerate(zip(pack.lens_host.tolist(), tl.tolist())):
        res.append(torch.nn.functional.ctc_loss(lp[lo: lo + n, None], targets[b: b + 1, :s].long(), torch.tensor([n]), torch.tensor([s]), blank=blank,
                                                reduction="none", zero_infinity=True))
        lo += n
    loss = torch.cat(res)
    return loss.detach(), torch.autograd.grad((loss * w.double()).sum(), [x])[0]


@gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lens,tlens,V,scale", [
    ([1, 2, 9, 17], [0, 1, 4, 8], 5, 2.0),              # one frame; a group of frames and one more
    ([120, 49, 150], [24, 24, 30], 1001, 10.0),         # one warp per recursion, and the first state of the second
    ([300, 260, 400], [125, 128, 65], 80, 40.0),        # several warps, widely different probabilities
    ([500, 31], [240, 15], 2049, 1.0),                  # four states per lane
    ([1300], [620], 37, 3.0),                           # eight
    ([40, 60], [7, 11], 33001, 2.0),                    # more vectors than a thread keeps; rows that start anywhere
    ([25, 30], [5, 9], 10240, 2.0),
])
def test_ctc_recursions_against_float64(lens, tlens, V, scale, dtype):
    """fp32 sums of a few hundred to a thousand products (2^-24 each, the exponent held apart): 2e-5; the bf16 gradient is rounded twice: 2^-8"""
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import ctc

    gen = torch.Generator("cuda").manual_seed(V)
    pack = PackInfo(torch.tensor(lens, dtype=torch.int32), torch.device("cuda"))
    targets = torch.randint(0, V - 1, (len(lens), max(tlens)), device="cuda", dtype=torch.int32, generator=gen)
    repeat = torch.rand(targets.shape, device="cuda", generator=gen) < 0.2
    targets[:, 1:] = torch.where(repeat[:, 1:], targets[:, :-1], targets[:, 1:])
    tl = torch.tensor(tlens, dtype=torch.int32)
    logits = (torch.randn(pack.n, V, device="cuda", generator=gen) * scale).to(dtype).requires_grad_(True)
    w = torch.rand(len(lens), device="cuda", generator=gen) + 0.5
    loss = ctc.ctc_loss_packed(logits, pack, targets, tl, blank_index=V - 1)
    (grad,) = torch.autograd.grad((loss * w).sum(), [logits])
    ref, ref_grad = _ctc_float64(logits, pack, targets, tl, V - 1, w)
    torch.testing.assert_close(loss.detach().double(), ref, atol=1e-4, rtol=2e-6)
    assert float((grad.double() - ref_grad).norm()) <= (2e-5 if dtype == torch.float32 else 2.0 ** -8) * float(ref_grad.norm())
    with torch.no_grad():
        assert torch.equal(ctc.ctc_loss_packed(logits.detach(), pack, targets, tl, blank_index=V - 1), loss.detach())


@gpu
@pytest.mark.parametrize("value", [float("-inf"), -3.0e38, -1e9, -1e5])
def test_ctc_masked_classes(value):
    """classes masked by -inf or a large negative number: not in the labels, and in them (the second sequence then has no alignment, or a huge loss)"""
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import ctc

    gen = torch.Generator("cuda").manual_seed(1)
    pack = PackInfo(torch.tensor([12, 9, 20], dtype=torch.int32), torch.device("cuda"))
    logits = torch.randn(pack.n, 30, device="cuda", generator=gen)
    logits[:, 21:25] = value
    targets = torch.randint(0, 20, (3, 4), device="cuda", dtype=torch.int32, generator=gen)
    tl = torch.tensor([4, 3, 2], dtype=torch.int32)
    for label in (None, 22):
        if label is not None:
            targets[1, 1] = label
        x = logits.clone().requires_grad_(True)
        loss = ctc.ctc_loss_packed(x, pack, targets, tl, blank_index=29)
        (grad,) = torch.autograd.grad(loss.sum(), [x])
        # log_softmax of -inf has no gradient: e^-1e5 is 0 in 64 bits as well
        ref, ref_grad = _ctc_float64(torch.clamp(x, min=-1e5) if value == float("-inf") else x, pack, targets, tl, 29, torch.ones(3, device="cuda"))
        if value == float("-inf") and label is not None:
            ref[1] = 0.0
        torch.testing.assert_close(loss.detach().double(), ref, atol=1e-4, rtol=1e-6)
        rows = slice(0, 12) if label is not None else slice(0, pack.n)  # a loss of 1e9 has no digits left for the alignment
        torch.testing.assert_close(grad[rows].double(), ref_grad[rows], atol=1e-5, rtol=0)
        assert bool(torch.isfinite(grad).all())
        if label is not None and value == float("-inf"):
            assert float(loss[1].detach()) == 0.0 and float(grad[12:21].abs().max()) == 0.0


@gpu
@pytest.mark.parametrize("dtype,V", [(torch.float32, 30), (torch.bfloat16, 30), (torch.bfloat16, 5003)])
@pytest.mark.parametrize("value", [None, -1e9, -1e10, -1e30])
def test_ctc_frames_filled_with_the_lowest_value(dtype, V, value):
    """
    or another large number: a frame without information, every class equally likely. (Its log(V) is below the resolution of 32 bits at that size:
    the loss is short of it)
    """
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import ctc

    gen = torch.Generator("cuda").manual_seed(V)
    pack = PackInfo(torch.tensor([12, 20], dtype=torch.int32), torch.device("cuda"))
    logits = torch.randn(pack.n, V, device="cuda", generator=gen).to(dtype)
    value = torch.finfo(dtype).min if value is None else value
    logits[5] = value
    logits[14] = -value
    logits[15, 1:] = value
    targets = torch.randint(1, 20, (2, 4), device="cuda", dtype=torch.int32, generator=gen)
    targets[1, 0] = 0  # frame 15 allows nothing else
    tl = torch.tensor([4, 3], dtype=torch.int32)
    x = logits.requires_grad_(True)
    loss = ctc.ctc_loss_packed(x, pack, targets, tl, blank_index=V - 1)
    (grad,) = torch.autograd.grad(loss.sum(), [x])
    flat = logits.detach().float().clone()
    flat[5], flat[14], flat[15, 1:] = 0.0, 0.0, -1e4
    ref, ref_grad = _ctc_float64(flat, pack, targets, tl, V - 1, torch.ones(2, device="cuda"))
    torch.testing.assert_close(loss.detach().double(), ref - math.log(V), atol=1e-4, rtol=1e-5)
    # frame 15 takes the second sequence through log space: 2^-24 of a loss of about 100 per frame, 20 frames
    tol = 1e-4 if dtype == torch.float32 else 2.0 ** -8
    assert float((grad.double() - ref_grad).norm()) <= tol * float(ref_grad.norm())


@gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("V", [9, 1000, 10001])
def test_ctc_rows_of_infeasible_sequences_are_cleared(V, dtype):
    """whole rows, wherever they start, and no others"""
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import ctc

    gen = torch.Generator("cuda").manual_seed(V)
    pack = PackInfo(torch.tensor([9, 3, 7], dtype=torch.int32), torch.device("cuda"))
    x = torch.randn(pack.n, V, device="cuda", generator=gen).to(dtype).requires_grad_(True)
    targets = torch.randint(0, V - 1, (3, 5), device="cuda", dtype=torch.int32, generator=gen)
    grads = []
    for tl in ([4, 5, 3], [4, 1, 3]):  # five labels in three frames
        loss = ctc.ctc_loss_packed(x, pack, targets, torch.tensor(tl, dtype=torch.int32), blank_index=V - 1)
        grads.append(torch.autograd.grad(loss.sum(), [x])[0])
        assert (float(loss[1].detach()) == 0.0) == (tl[1] == 5)
    assert not grads[0][9:12].any() and bool(grads[1][9:12].any(1).all())
    assert torch.equal(grads[0][:9], grads[1][:9]) and torch.equal(grads[0][12:], grads[1][12:])


@gpu
@pytest.mark.parametrize("lens,tlens,V", [([40, 1, 7], [9, 0, 3], 50), ([300, 260], [125, 128], 80), ([500, 31], [240, 15], 300), ([1300], [620], 37)])
def test_ctc_recursions_in_log_space_against_float64(lens, tlens, V):
    """
    a label masked by a large finite number in the first frames, which the alignments can do without: every sequence takes the recursions in log
    space. There a sum is rounded to 2^-24 of the loss per frame, and these errors add up like a random walk: 2^-24 * sqrt(frames) * loss
    """
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import ctc

    gen = torch.Generator("cuda").manual_seed(V)
    pack = PackInfo(torch.tensor(lens, dtype=torch.int32), torch.device("cuda"))
    targets = torch.randint(0, V - 2, (len(lens), max(tlens)), device="cuda", dtype=torch.int32, generator=gen)
    repeat = torch.rand(targets.shape, device="cuda", generator=gen) < 0.2
    targets[:, 1:] = torch.where(repeat[:, 1:], targets[:, :-1], targets[:, 1:])
    logits = torch.randn(pack.n, V, device="cuda", generator=gen) * 2
    lo = 0
    for b, (n, s) in enumerate(zip(lens, tlens)):
        if s:
            targets[b, s - 1] = V - 2  # the last label, nowhere else: masked in a frame that is too early for it
            logits[lo, V - 2] = -1e9
        lo += n
    x = logits.requires_grad_(True)
    tl = torch.tensor(tlens, dtype=torch.int32)
    loss = ctc.ctc_loss_packed(x, pack, targets, tl, blank_index=V - 1)
    (grad,) = torch.autograd.grad(loss.sum(), [x])
    ref, ref_grad = _ctc_float64(x, pack, targets, tl, V - 1, torch.ones(len(lens), device="cuda"))
    torch.testing.assert_close(loss.detach().double(), ref, atol=1e-4, rtol=4 * max(lens) ** 0.5 * 2.0 ** -24)
    bound = 8 * max(lens) ** 0.5 * 2.0 ** -24 * float(ref.max()) + 2e-5
    assert float((grad.double() - ref_grad).norm()) <= bound * float(ref_grad.norm())
    with torch.no_grad():  # broken input stays visible there
        for value in (float("nan"), float("inf")):
            y = logits.detach().clone()
            y[lens[0] // 2, V - 1] = value
            assert bool(torch.isnan(ctc.ctc_loss_packed(y, pack, targets, tl, blank_index=V - 1)[0]))
