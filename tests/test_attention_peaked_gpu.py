"""
Attention forward kernels on rows with few large probabilities. The kernels round the probabilities of a row to 16 bits relative to the row's maximum up
to there, so the largest weight is 1 and exact; the sums are in 32 bits. The oracle is that algorithm in 64 bits (tiles of 64 keys, weights rounded):
its error against the definition is what the rounding of the weights costs, and the kernel's may be no more than that; 8 % are allowed for its sums and
exponentials in 32 bits and for single values that round the other way. Weights relative to a maximum that lags behind have 1.1 to 1.25 times the error.
"""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _bf(x):
    return x.float().to(torch.bfloat16).double()


def _err(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


def _tiled(s, v, keep=None, scale=1.0):
    """softmax(s) v over tiles of 64 keys: s [H, Tq, Tk] (-inf: hidden), v [H, Tk, D] in 64 bits; keep: dropout decisions, kept weights times scale"""
    m = torch.full(s.shape[:2] + (1,), float("-inf"), dtype=s.dtype, device=s.device)
    den, out = torch.zeros_like(m), torch.zeros(s.shape[:2] + v.shape[-1:], dtype=s.dtype, device=s.device)
    for j in range(0, s.shape[2], 64):
        t = s[..., j: j + 64]
        to = torch.maximum(m, t.amax(-1, keepdim=True))
        corr = torch.exp(m - to)
        e = torch.exp(t - to)
        m, den = to, den * corr + e.sum(-1, keepdim=True)
        if keep is not None:
            e = e * keep[..., j: j + 64] * scale
        out = out * corr + _bf(e) @ v[:, j: j + 64]
    return out / den


@pytest.mark.parametrize("factor", [1.0, 4.0, 8.0])
@pytest.mark.parametrize("T,causal,offset", [(512, False, 0.0), (512, False, 24.0), (300, True, 0.0), (129, False, 0.0)])
def test_sdpa_peaked_rows(T, causal, offset, factor):
    from returnn_b200.ops import sdpa as S

    g = torch.Generator(device="cuda").manual_seed(3)
    H, D = 4, 64
    rand = lambda: torch.randn(1, T, H, D, generator=g, device="cuda")  # noqa: E731
    q, k, v, dy = ((rand() * factor).to(torch.bfloat16), (rand() + offset / 6).to(torch.bfloat16), (rand() + offset).to(torch.bfloat16), rand().to(torch.bfloat16))
    x = [t.clone().requires_grad_(True) for t in (q, k, v)]
    got = S.sdpa_heads(*x, causal=causal)
    got_dq = torch.autograd.grad(got, x[:1], dy)[0][0].transpose(0, 1)
    got = got.detach()[0].transpose(0, 1)
    q, k, v, dy = (t[0].transpose(0, 1).double() for t in (q, k, v, dy))
    s = (q @ k.transpose(1, 2)) * 0.125
    if causal:
        s = s.masked_fill(~torch.ones(T, T, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    p = torch.softmax(s, -1)
    want, out = p @ v, _tiled(s, v)
    assert _err(got, want) <= 1.08 * _err(_bf(out), want), (_err(got, want), _err(_bf(out), want))
    # the query gradient: dS = P (dP - dO . O) from the output before its rounding, dS in 16 bits
    dp = dy @ v.transpose(1, 2)
    grad = lambda o, rnd: rnd(rnd(p * (dp - (dy * o).sum(-1, keepdim=True))) @ k * 0.125)  # noqa: E731
    want, out = grad(want, lambda t: t), grad(out, _bf)
    assert _err(got_dq, want) <= 1.08 * _err(out, want), (_err(got_dq, want), _err(out, want))


@pytest.mark.parametrize("factor", [1.0, 4.0])
@pytest.mark.parametrize("Tq,Tk", [(300, 300), (70, 190), (128, 64)])
def test_sdpa_peaked_rows_with_dropout(Tq, Tk, factor):
    from returnn_b200.ops import sdpa as S
    from returnn_b200.ops.elementwise import _seed_tensor

    g = torch.Generator(device="cuda").manual_seed(4)
    H, D, p = 4, 64, 0.25
    rand = lambda t: torch.randn(1, t, H, D, generator=g, device="cuda")  # noqa: E731
    q, k, v = (rand(Tq) * factor).to(torch.bfloat16), rand(Tk).to(torch.bfloat16), rand(Tk).to(torch.bfloat16)
    seed = _seed_tensor(q.device)
    state = seed.clone()
    keep = torch.zeros(H, Tq, Tk, dtype=torch.double, device="cuda")
    for j in range(0, Tk, D):  # the decisions: with no scores and the identity on a block of keys as values the output is the kept weights
        n = min(D, Tk - j)
        block = torch.zeros(1, Tk, H, D, device="cuda", dtype=torch.bfloat16)
        block[0, j: j + n, :, :n] = torch.eye(n, device="cuda", dtype=torch.bfloat16)[:, None]
        seed.copy_(state)
        keep[..., j: j + n] = (S.sdpa_heads(q * 0, k, block, dropout_p=p)[0, :, :, :n] > 0).transpose(0, 1).double()
    seed.copy_(state)
    got = S.sdpa_heads(q, k, v, dropout_p=p)[0].transpose(0, 1)
    q, k, v = (t[0].transpose(0, 1).double() for t in (q, k, v))
    s = (q @ k.transpose(1, 2)) * 0.125
    want, out = (torch.softmax(s, -1) * keep / (1 - p)) @ v, _tiled(s, v, keep, 1 / (1 - p))
    assert _err(got, want) <= 1.08 * _err(_bf(out), want), (_err(got, want), _err(_bf(out), want))


@pytest.mark.parametrize("factor", [1.0, 4.0, 8.0])
@pytest.mark.parametrize("T", [129, 300, 512])
def test_rel_pos_peaked_rows(T, factor):
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import attention_native as an

    g = torch.Generator(device="cuda").manual_seed(5)
    H, D = 4, 64
    pack = PackInfo(torch.tensor([T], dtype=torch.int32), torch.device("cuda"))
    qkv = torch.randn(T, H, 3, D, generator=g, device="cuda") * torch.tensor([factor, 1.0, 1.0], device="cuda")[:, None]
    qkv = qkv.to(torch.bfloat16)
    pos = (torch.randn(2 * T - 1, H * D, generator=g, device="cuda") * 0.5).to(torch.bfloat16)
    zero = torch.zeros(H, D, device="cuda")
    # (with gradients: the kernel of the training pass)
    x = qkv.reshape(T, -1).clone().requires_grad_(True)
    got = an.rel_pos_attention_packed(x, pos, zero, zero, pack, num_heads=H, head_dim=D, scale=0.125).detach().view(T, H, D).transpose(0, 1)
    q, k, v = (qkv[:, :, i].transpose(0, 1).double() for i in range(3))
    band = q @ pos.double().view(-1, H, D).permute(1, 2, 0)
    at = torch.arange(T, device="cuda")
    s = (q @ k.transpose(1, 2) + torch.gather(band, 2, (at[None] - at[:, None] + T - 1).expand(H, T, T))) * 0.125
    want = torch.softmax(s, -1) @ v
    # two groups of 64 keys of each 128, each with a maximum of its own, merged at the end: a maximum of either kind is never behind the group's
    half = (at // 64 % 2).bool()
    parts = []
    for sel in (~half, half):
        sp = s[..., sel]
        parts.append((torch.logsumexp(sp, -1, keepdim=True), _tiled(sp, v[:, sel])))
    lse = torch.logsumexp(torch.cat([a for a, _ in parts], -1), -1, keepdim=True)
    out = sum(torch.exp(a - lse) * o for a, o in parts)
    assert _err(got, want) <= 1.08 * _err(_bf(out), want), (_err(got, want), _err(_bf(out), want))
