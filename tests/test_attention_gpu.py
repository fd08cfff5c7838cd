"""
Packed relative-position attention (batched tcgen05 GEMMs + softmax kernels) against the fp32 torch math.
"""

import pytest
import torch

gpu = pytest.mark.gpu


def _reference(qkv, pos, u, v, pack, H, D, scale):
    from returnn_b200.ops import attention as att

    N = qkv.shape[0]
    x = qkv.reshape(N, H, 3, D)
    pad = pack.unpack(x)
    T = pad.shape[1]
    q = pad[:, :, :, 0].permute(0, 2, 1, 3)
    k = pad[:, :, :, 1].permute(0, 2, 1, 3)
    vv = pad[:, :, :, 2].permute(0, 2, 1, 3)
    L = (pos.shape[0] + 1) // 2
    p = pos.reshape(2 * L - 1, H, D).permute(1, 0, 2)
    if T != L:
        p = p[:, (L - 1) - (T - 1): (L - 1) + T]
    out = att.rel_pos_attention_reference(q, k, vv, p, u, v, pack.lens, scale=scale)
    out = out.permute(0, 2, 1, 3).reshape(out.shape[0], T, H * D)
    return pack.pack(out)


@gpu
@pytest.mark.parametrize("lens,H,D", [([5], 1, 64), ([130, 64, 1, 77], 4, 64), ([334, 200, 129], 8, 64), ([40, 33], 2, 128)])
def test_rel_pos_attention_packed(lens, H, D):
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import attention_native as an, gemm

    torch.manual_seed(0)
    lens_t = torch.tensor(lens, dtype=torch.int32)
    pack = PackInfo(lens_t, torch.device("cuda"))
    N, L = pack.n, pack.max_len
    assert an.supports_packed(H, D, L)
    qkv = (torch.randn(N, H * 3 * D, device="cuda") * 0.7).to(torch.bfloat16).requires_grad_(True)
    pos = (torch.randn(2 * L - 1, H * D, device="cuda") * 0.7).to(torch.bfloat16).requires_grad_(True)
    u = (torch.randn(H, D, device="cuda") * 0.3).requires_grad_(True)
    v = (torch.randn(H, D, device="cuda") * 0.3).requires_grad_(True)
    d_out = torch.randn(N, H * D, device="cuda").to(torch.bfloat16)
    scale = D ** -0.5
    out = an.rel_pos_attention_packed(qkv, pos, u, v, pack, num_heads=H, head_dim=D, scale=scale, dropout_p=0.0)
    out.backward(d_out)
    gemm.check_status()
    q32 = qkv.detach().float().requires_grad_(True)
    p32 = pos.detach().float().requires_grad_(True)
    u32 = u.detach().clone().requires_grad_(True)
    v32 = v.detach().clone().requires_grad_(True)
    ref = _reference(q32, p32, u32, v32, pack, H, D, scale)
    ref.backward(d_out.float())
    torch.testing.assert_close(out.float(), ref, atol=3e-2, rtol=3e-2)
    torch.testing.assert_close(qkv.grad.float(), q32.grad, atol=6e-2, rtol=5e-2)
    torch.testing.assert_close(pos.grad.float(), p32.grad, atol=0.15, rtol=5e-2)
    torch.testing.assert_close(u.grad, u32.grad, atol=0.3, rtol=5e-2)
    torch.testing.assert_close(v.grad, v32.grad, atol=0.3, rtol=5e-2)


@gpu
def test_rel_pos_attention_dropout_consistent():
    """with dropout: forward mean is preserved and backward uses the mask of its forward (finite differences on a linear probe)"""
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import attention_native as an

    torch.manual_seed(1)
    H, D = 2, 64
    pack = PackInfo(torch.tensor([70, 50], dtype=torch.int32), torch.device("cuda"))
    N, L = pack.n, pack.max_len
    qkv = (torch.randn(N, H * 3 * D, device="cuda") * 0.5).to(torch.bfloat16)
    pos = (torch.randn(2 * L - 1, H * D, device="cuda") * 0.5).to(torch.bfloat16)
    outs = [an.rel_pos_attention_packed(qkv, pos, None, None, pack, num_heads=H, head_dim=D, scale=D ** -0.5, dropout_p=0.3).float() for _ in range(64)]
    base = an.rel_pos_attention_packed(qkv, pos, None, None, pack, num_heads=H, head_dim=D, scale=D ** -0.5, dropout_p=0.0).float()
    mean = torch.stack(outs).mean(0)
    assert (mean - base).abs().mean() < 0.05
    assert (outs[0] - outs[1]).abs().max() > 1e-3


@gpu
@pytest.mark.parametrize("lens,H,extra", [([1], 1, 0), ([64, 63, 65], 3, 0), ([128, 129, 127, 2], 2, 5), ([512, 300], 1, 0), ([257, 256], 4, 1)])
def test_rel_pos_attention_head_dim_64_tile_edges(lens, H, extra):
    """lengths around the tiles of 64 keys and 128 queries, a position table that is longer than the batch needs"""
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import attention_native as an, gemm

    torch.manual_seed(len(lens) + H)
    D = 64
    pack = PackInfo(torch.tensor(lens, dtype=torch.int32), torch.device("cuda"))
    L = min(pack.max_len + extra, (pack.max_len + 63) // 64 * 64)
    qkv = torch.randn(pack.n, H * 3 * D, device="cuda").to(torch.bfloat16).requires_grad_(True)
    pos = torch.randn(2 * L - 1, H * D, device="cuda").to(torch.bfloat16).requires_grad_(True)
    u = (torch.randn(H, D, device="cuda") * 0.3).requires_grad_(True)
    v = (torch.randn(H, D, device="cuda") * 0.3).requires_grad_(True)
    dy = torch.randn(pack.n, H * D, device="cuda").to(torch.bfloat16)
    out = an.rel_pos_attention_packed(qkv, pos, u, v, pack, num_heads=H, head_dim=D, scale=0.125)
    got = [out, *torch.autograd.grad(out, [qkv, pos, u, v], dy)]
    gemm.check_status()
    x = [t.detach().double().requires_grad_(True) for t in (qkv, pos, u, v)]
    ref = _reference(*x, pack, H, D, 0.125)
    want = [ref, *torch.autograd.grad(ref, x, dy.double())]
    for a, b in zip(got, want):
        # bf16 operands, probabilities and score gradients: 2^-9 each
        assert (a.double() - b).norm() <= 1.2e-2 * b.norm() + 1e-3


@gpu
def test_rel_pos_attention_head_dim_64_dropout_gradients():
    """with the identity as values the output is the dropped probabilities: they give the mask, which the backward pass has to use as well"""
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import attention_native as an
    from returnn_b200.ops.elementwise import _seed_tensor

    torch.manual_seed(3)
    T, H, D, p = 64, 2, 64, 0.25
    pack = PackInfo(torch.tensor([T], dtype=torch.int32), torch.device("cuda"))
    qkv = torch.randn(T, H, 3, D, device="cuda").to(torch.bfloat16)
    pos = torch.randn(2 * T - 1, H * D, device="cuda").to(torch.bfloat16)
    eye = qkv.clone()
    eye[:, :, 2] = torch.eye(T, device="cuda", dtype=torch.bfloat16)[:, None]
    seed = _seed_tensor(qkv.device)
    state = seed.clone()
    run = lambda x, ps: an.rel_pos_attention_packed(x.reshape(T, -1), ps, None, None, pack, num_heads=H, head_dim=D, scale=0.125, dropout_p=p)  # noqa: E731
    mask = (run(eye, pos).view(T, H, T).transpose(0, 1) > 0).double()
    assert abs(mask.mean().item() - (1 - p)) < 0.03
    seed.copy_(state)
    x, ps = qkv.clone().requires_grad_(True), pos.clone().requires_grad_(True)
    dy = torch.randn(T, H * D, device="cuda").to(torch.bfloat16)
    got = torch.autograd.grad(run(x, ps), [x, ps], dy)
    xr, pr = qkv.double().requires_grad_(True), pos.double().requires_grad_(True)
    q, k, v = (xr[:, :, i].transpose(0, 1) for i in range(3))
    band = q @ pr.view(-1, H, D).permute(1, 2, 0)
    at = torch.arange(T, device="cuda")
    s = (q @ k.transpose(1, 2) + torch.gather(band, 2, (at[None] - at[:, None] + T - 1).expand(H, T, T))) * 0.125
    out = ((torch.softmax(s, -1) * mask / (1 - p)) @ v).transpose(0, 1).reshape(T, -1)
    for a, b in zip(got, torch.autograd.grad(out, [xr, pr], dy.double())):
        assert (a.double() - b).norm() <= 1.2e-2 * b.norm()
