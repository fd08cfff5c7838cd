"""Attention gradients of short sequences (one kernel up to 128 queries and keys) at the edges of its range, against 64 bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _exact(q, k, v, k_lens, causal, dy):
    q, k, v = (x.detach().double().requires_grad_(True) for x in (q, k, v))
    Tq, Tk = q.shape[1], k.shape[1]
    s = torch.einsum("bihd,bjhd->bhij", q, k) * 0.125
    ok = torch.ones(q.shape[0], 1, Tq, Tk, dtype=torch.bool, device="cuda")
    if k_lens is not None:
        ok = ok & (torch.arange(Tk, device="cuda")[None, None, None] < k_lens[:, None, None, None])
    if causal:
        ok = ok & (torch.arange(Tk, device="cuda")[None, :] <= torch.arange(Tq, device="cuda")[:, None] + (Tk - Tq))[None, None]
    p = torch.softmax(s.masked_fill(~ok, -1e30), -1) * ok
    y = torch.einsum("bhij,bjhd->bihd", p, v)
    return [y.detach(), *torch.autograd.grad(y, [q, k, v], dy.double())]


@pytest.mark.parametrize("Tq,Tk", [(1, 1), (1, 128), (128, 1), (16, 17), (64, 64), (65, 127), (127, 65), (128, 128), (128, 129)])
@pytest.mark.parametrize("causal,lens", [(False, None), (True, None), (False, (0, 1.0, 0.3)), (True, (1.0, 0.5, 0))])
def test_short_sequences(Tq, Tk, causal, lens):
    from returnn_b200.ops import gemm, guard
    from returnn_b200.ops.sdpa import sdpa_heads

    B, H = 3, 2
    g = torch.Generator(device="cuda").manual_seed(Tq * 1000 + Tk)
    rnd = lambda t: torch.randn(B, t, H, 64, generator=g, device="cuda").bfloat16()  # noqa: E731
    q, k, v, dy = rnd(Tq), rnd(Tk), rnd(Tk), rnd(Tq)
    kl = None if lens is None else torch.tensor([int(x * Tk) for x in lens], dtype=torch.int32, device="cuda")
    want = _exact(q, k, v, kl, causal, dy)
    if kl is not None:  # padding from the next step of 16 keys on may be anything (the tiles of the forward pass are 64 keys)
        for b, n in enumerate(kl.tolist()):
            k[b, -(-n // 64) * 64:] = float("nan")
            v[b, -(-n // 64) * 64:] = float("nan")
    leaves = [x.requires_grad_(True) for x in (q, k, v)]
    with guard.CanaryAllocations() as canary:
        y = sdpa_heads(*leaves, k_lens=kl, causal=causal)
        got = [y.detach(), *torch.autograd.grad(y, leaves, dy)]
    canary.check()
    gemm.check_status()
    for a, b in zip(got, want):
        # operands P and dS and the results are rounded to bf16 (2^-9 each); sums of both signs of up to 128 of them
        assert float((a.double() - b).norm()) <= 2e-2 * float(b.norm()) + 1e-4


@pytest.mark.parametrize("Tq,Tk", [(31, 31), (128, 128), (17, 128), (128, 65)])
def test_dropout_decisions_are_those_of_the_forward_pass(Tq, Tk):
    """
    The decisions, read out of the forward pass (with the identity on a block of keys as values its output is the kept probabilities), and all
    gradients against the definition with them in 64 bits.
    """
    from returnn_b200.ops.elementwise import _seed_tensor
    from returnn_b200.ops.sdpa import sdpa_heads

    g = torch.Generator(device="cuda").manual_seed(Tq + Tk)
    B, H, p = 2, 2, 0.3
    q, k, v, dy = ((torch.randn(B, t, H, 64, generator=g, device="cuda") * f).bfloat16().requires_grad_(True)
                   for t, f in ((Tq, 0.7), (Tk, 0.7), (Tk, 1.0), (Tq, 1.0)))
    seed = _seed_tensor(q.device)
    state = seed.clone()
    mask = torch.zeros(B, H, Tq, Tk, dtype=torch.double, device="cuda")
    for j in range(0, Tk, 64):
        n = min(64, Tk - j)
        block = torch.zeros(B, Tk, H, 64, dtype=torch.bfloat16, device="cuda")
        block[:, j: j + n, :, :n] = torch.eye(n, device="cuda", dtype=torch.bfloat16)[:, None]
        seed.copy_(state)
        mask[..., j: j + n] = (sdpa_heads(q.detach(), k.detach(), block, dropout_p=p)[..., :n] > 0).transpose(1, 2).double()
    assert abs(float(mask.mean()) - (1 - p)) < 4 * (p * (1 - p) / mask.numel()) ** 0.5
    seed.copy_(state)
    y = sdpa_heads(q, k, v, dropout_p=p)
    got = torch.autograd.grad(y, [q, k, v], dy.detach())
    r = [t.detach().double().requires_grad_(True) for t in (q, k, v)]
    w = torch.softmax(torch.einsum("bihd,bjhd->bhij", r[0], r[1]) * 0.125, -1) * mask / (1 - p)
    want = torch.einsum("bhij,bjhd->bihd", w, r[2])
    for a, b in zip((y, *got), (want, *torch.autograd.grad(want, r, dy.detach().double()))):
        # probabilities, dS and results rounded to bf16, 2^-9 each; a decision that differs is an error of sqrt(1 / (1 - p)) of its element
        assert float((a.double() - b).detach().norm()) <= 1e-2 * float(b.detach().norm())


def test_common_offset_of_the_values():
    """the row sums of P * dP come from 32-bit values: an offset that all values share leaves the query gradient (see rb200_flash_fwd)"""
    from returnn_b200.ops.sdpa import sdpa_heads

    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda m: (torch.randn(2, 100, 2, 64, generator=g, device="cuda") + m).bfloat16().requires_grad_(True)  # noqa: E731
    q, k, v, dy = rnd(0.), rnd(4.), rnd(24.), rnd(0.)
    got = torch.autograd.grad(sdpa_heads(q, k, v), [q], dy)[0].double()
    want = _exact(q, k, v, None, False, dy.detach())[1]
    assert float((got - want).norm()) <= 0.3 * float(want.norm())
