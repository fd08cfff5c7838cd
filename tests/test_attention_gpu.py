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


@gpu
def test_rel_pos_attention_query_gradient_where_values_share_an_offset():
    """
    An offset common to all keys or all values leaves the query gradient as it is, as far as the row sums of P * dP are known: here
    24 |dO| = 24 * 8, where dS itself is 8 P. What remains is the 16-bit rounding of the n probabilities in the output,
    24 * 8 * 0.0009 / sqrt(n) per row, times the common key 4, against 8 / sqrt(n): 0.09 (row sums from the output in 16 bits: 1 to 2).
    """
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import attention_native as an

    torch.manual_seed(8)
    T, H, D = 300, 2, 64
    pack = PackInfo(torch.tensor([T], dtype=torch.int32), torch.device("cuda"))
    qkv = torch.randn(T, H, 3, D, device="cuda") * torch.tensor([0.02, 1.0, 1.0], device="cuda")[:, None]
    qkv = (qkv + torch.tensor([0.0, 4.0, 24.0], device="cuda")[:, None]).to(torch.bfloat16).reshape(T, -1)
    pos = (torch.randn(2 * T - 1, H * D, device="cuda") * 0.02).to(torch.bfloat16)
    u = torch.zeros(H, D, device="cuda")
    dy = torch.randn(T, H * D, device="cuda").to(torch.bfloat16)
    x = qkv.clone().requires_grad_(True)
    got = torch.autograd.grad(an.rel_pos_attention_packed(x, pos, u, u, pack, num_heads=H, head_dim=D, scale=0.125), x, dy)[0]
    xr = qkv.double().requires_grad_(True)
    want = torch.autograd.grad(_reference(xr, pos.double(), u.double(), u.double(), pack, H, D, 0.125), xr, dy.double())[0]
    got, want = (t.double().view(T, H, 3, D)[:, :, 0] for t in (got, want))
    assert (got - want).norm() <= 0.2 * want.norm(), ((got - want).norm() / want.norm()).item()


@gpu
@pytest.mark.parametrize("lens,H,p", [([150, 192, 40], 2, 0.0), ([150, 192, 40], 2, 0.25), ([321, 257], 1, 0.1), ([64, 1], 3, 0.1)])
def test_rel_flash_bwd_on_saved_probabilities(lens, H, p):
    """
    the form of the backward kernel that the encoder executor takes: probabilities, dropped probabilities and output as a forward pass left
    them; the score gradients, both query gradients and the band against the definition in 64 bits
    """
    import ctypes
    from returnn_b200.ops import _lib, gemm as G

    torch.manual_seed(len(lens) + H)
    dev, B, L = "cuda", len(lens), max(lens)
    Lp, HD, scale = (L + 63) // 64 * 64, H * 64, 0.125
    R = 2 * L - 1
    bf = lambda *s: torch.randn(*s, device=dev).to(torch.bfloat16)  # noqa: E731
    valid = (torch.arange(Lp, device=dev)[None] < torch.tensor(lens, device=dev)[:, None])
    qu, qv, k, v, do = (bf(B, Lp, HD) * valid[:, :, None] for _ in range(5))
    pos = bf(R, HD)
    heads = lambda t: t.view(B, -1, H, 64).transpose(1, 2).double()  # noqa: E731
    ok = valid[:, None, :, None] & valid[:, None, None, :]
    at = torch.arange(Lp, device=dev)
    rel = L - 1 + at[None] - at[:, None]  # position row of (query, key)
    inside = (rel >= 0) & (rel < R)
    posh = pos.view(R, H, 64).transpose(0, 1).double()
    s = heads(qu) @ heads(k).transpose(2, 3)
    s = s + torch.gather(heads(qv) @ posh.transpose(1, 2), 3, rel.clamp(0, R - 1).expand(B, H, Lp, Lp))
    w = torch.nan_to_num(torch.softmax((s * scale).masked_fill(~ok, float("-inf")), -1)).to(torch.bfloat16)
    keep = (torch.rand(B, H, Lp, Lp, device=dev) >= p).double()
    wd = (w.double() * keep / (1 - p)).to(torch.bfloat16)
    o = (wd.double() @ heads(v)).transpose(1, 2).reshape(B, Lp, HD).float()
    # the definition
    dp = heads(do) @ heads(v).transpose(2, 3) * keep / (1 - p)
    ds = w.double() * (dp - (heads(do) * heads(o)).sum(-1, keepdim=True))
    dqu = ds @ heads(k) * scale
    band = torch.zeros(B, H, Lp, R, device=dev, dtype=torch.float64).scatter_add(3, rel.clamp(0, R - 1).expand(B, H, Lp, Lp), ds * inside)
    dqv = band @ posh * scale
    # the kernel
    geo = (ctypes.c_int * 2)()
    vp, i32, f32 = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
    _lib.check(_lib.bind("rb200_rel_flash_band", [i32, i32, vp, vp])(Lp, L - 1, ctypes.addressof(geo), ctypes.addressof(geo) + 4), "band")
    got_qu, got_qv = (torch.zeros(B, Lp, HD, device=dev, dtype=torch.bfloat16) for _ in range(2))
    got_band = torch.zeros(H, B, Lp, geo[1], device=dev, dtype=torch.bfloat16)
    got_ds = torch.zeros(B, H, Lp, Lp, device=dev, dtype=torch.bfloat16)
    lens_t = torch.tensor(lens, dtype=torch.int32, device=dev)
    fn = _lib.bind("rb200_rel_flash_bwd", [vp] * 16 + [i32] * 5 + [f32, f32, vp, vp])
    _lib.check(fn(qu.data_ptr(), qv.data_ptr(), k.data_ptr(), v.data_ptr(), pos.data_ptr(), o.data_ptr(), do.data_ptr(), got_qu.data_ptr(),
                  got_qv.data_ptr(), w.data_ptr(), wd.data_ptr(), got_ds.data_ptr(), got_band.data_ptr(), None, None, lens_t.data_ptr(), B, H, Lp, R, L - 1,
                  scale, p, G.status_tensor(lens_t.device).data_ptr(), _lib.stream_ptr()), "rel_flash_bwd")
    G.check_status()
    unheads = lambda t: t.transpose(1, 2).reshape(B, Lp, HD)  # noqa: E731
    for got, want in ((got_ds, ds), (got_band[..., geo[0]: geo[0] + R].transpose(0, 1), band), (got_qu, unheads(dqu)), (got_qv, unheads(dqv))):
        # dS is rounded to bf16 (2^-9), the query gradients once more
        assert (got.double() - want).norm() <= 2 * 2 ** -9 * want.norm() + 1e-6


@gpu
def test_rel_pos_attention_gradients_are_the_same_in_every_run():
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import attention_native as an

    torch.manual_seed(2)
    H, D = 4, 64
    pack = PackInfo(torch.tensor([300, 257, 40] * 4, dtype=torch.int32), torch.device("cuda"))
    x = [torch.randn(*s, device="cuda").to(dt).requires_grad_(True) for s, dt in (
        ((pack.n, H * 3 * D), torch.bfloat16), ((599, H * D), torch.bfloat16), ((H, D), torch.float32), ((H, D), torch.float32))]
    dy = torch.randn(pack.n, H * D, device="cuda").to(torch.bfloat16)
    runs = [torch.autograd.grad(an.rel_pos_attention_packed(*x, pack, num_heads=H, head_dim=D, scale=0.125), x, dy) for _ in range(8)]
    for r in runs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(r, runs[0]))


@gpu
@pytest.mark.parametrize("D,T", [(64, 270), (64, 150), (128, 200)])
def test_rel_pos_attention_dropout_gradients_over_several_tiles(D, T):
    """the decisions of all tiles, read out block by block: with the identity on a block of keys as values the output is the kept probabilities"""
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import attention_native as an
    from returnn_b200.ops.elementwise import _seed_tensor

    torch.manual_seed(9)
    H, p = 2, 0.2
    lens = [T, 40]
    pack = PackInfo(torch.tensor(lens, dtype=torch.int32), torch.device("cuda"))
    qkv = (torch.randn(pack.n, H, 3, D, device="cuda") * 0.7).to(torch.bfloat16)
    pos = (torch.randn(2 * T - 1, H * D, device="cuda") * 0.7).to(torch.bfloat16)
    seed = _seed_tensor(qkv.device)
    state = seed.clone()

    def run(x, ps):
        seed.copy_(state)
        return an.rel_pos_attention_packed(x.reshape(pack.n, -1), ps, None, None, pack, num_heads=H, head_dim=D, scale=D ** -0.5, dropout_p=p)

    mask = torch.zeros(H, T, T, device="cuda", dtype=torch.float64)
    for j in range(0, T, D):
        x, n = qkv.clone(), min(D, T - j)
        x[:, :, 2] = 0
        x[j: j + n, :, 2, :n] = torch.eye(n, device="cuda", dtype=torch.bfloat16)[:, None]
        mask[..., j: j + n] = (run(x, pos)[:T].view(T, H, D)[..., :n] > 0).transpose(0, 1).double()
    assert abs(mask.mean().item() - (1 - p)) < 0.02
    x, ps = qkv.clone().requires_grad_(True), pos.clone().requires_grad_(True)
    dy = torch.randn(pack.n, H * D, device="cuda").to(torch.bfloat16)
    dy[T:] = 0  # (the second sequence only shares the launch)
    got = torch.autograd.grad(run(x, ps), [x, ps], dy)
    xr, pr = qkv[:T].double().requires_grad_(True), pos.double().requires_grad_(True)
    q, k, v = (xr[:, :, i].transpose(0, 1) for i in range(3))
    band = q @ pr.view(-1, H, D).permute(1, 2, 0)
    at = torch.arange(T, device="cuda")
    s = (q @ k.transpose(1, 2) + torch.gather(band, 2, (at[None] - at[:, None] + T - 1).expand(H, T, T))) * D ** -0.5
    out = ((torch.softmax(s, -1) * mask / (1 - p)) @ v).transpose(0, 1).reshape(T, -1)
    for a, b in zip((got[0][:T], got[1]), torch.autograd.grad(out, [xr, pr], dy[:T].double())):
        assert (a.double() - b).norm() <= 1.2e-2 * b.norm()
    assert float(got[0][T:].abs().max()) == 0.0


@gpu
@pytest.mark.parametrize("lens,H", [([150, 192, 40], 2), ([64, 1], 1), ([65, 129, 0, 320], 3), ([512], 1)])
@pytest.mark.parametrize("saved", [True, False])
def test_rel_flash_bwd_writes_the_padding(lens, H, saved):
    """buffers full of NaN come back with the values of zeroed ones: every column and row that no tile of keys fills is written as zero"""
    import ctypes
    from returnn_b200.ops import _lib, gemm as G

    dev, bf, HD, B, L = "cuda", torch.bfloat16, H * 64, len(lens), max(lens)
    Lp, R = (L + 63) // 64 * 64, 2 * L - 1
    torch.manual_seed(5)
    lens_t = torch.tensor(lens, dtype=torch.int32, device=dev)
    valid = (torch.arange(Lp, device=dev)[None] < lens_t[:, None])
    qu, qv, k, v, do = ((torch.randn(B, Lp, HD, device=dev) * valid[..., None]).to(bf) for _ in range(5))
    pos, o = torch.randn(R, HD, device=dev).to(bf), torch.randn(B, Lp, HD, device=dev)
    w = torch.rand(B, H, Lp, Lp, device=dev).to(bf) * 0.01
    lse = torch.full((B, H, Lp), 12.0, device=dev)
    vp, i32, f32 = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
    geo = (ctypes.c_int * 2)()
    _lib.check(_lib.bind("rb200_rel_flash_band", [i32, i32, vp, vp])(Lp, L - 1, ctypes.addressof(geo), ctypes.addressof(geo) + 4), "band")
    fn = _lib.bind("rb200_rel_flash_bwd", [vp] * 16 + [i32] * 5 + [f32, f32, vp, vp])
    res = []
    for fill in (0.0, float("nan")):
        dqu, dqv, band = (torch.full(s, fill, device=dev, dtype=bf) for s in ((B, Lp, HD), (B, Lp, HD), (H, B, Lp, geo[1])))
        pw, ds = w.clone(), torch.zeros(B, H, Lp, Lp, device=dev, dtype=bf)
        _lib.check(fn(qu.data_ptr(), qv.data_ptr(), k.data_ptr(), v.data_ptr(), pos.data_ptr(), o.data_ptr(), do.data_ptr(), dqu.data_ptr(), dqv.data_ptr(),
                      w.data_ptr() if saved else None, pw.data_ptr(), ds.data_ptr(), band.data_ptr(), lse.data_ptr(), None, lens_t.data_ptr(), B, H, Lp, R,
                      L - 1, 0.125, 0.0, G.status_tensor(lens_t.device).data_ptr(), _lib.stream_ptr()), "rel_flash_bwd")
        G.check_status()
        res.append((dqu, dqv, band))
    for a, b in zip(*res):
        assert torch.isfinite(b).all() and torch.equal(a, b)
    dqu, dqv, band = res[1]
    assert not dqu[~valid].any() and not dqv[~valid].any() and not band[:, ~valid].any()
    # row i of the band holds dS[i, j] at column center + j - i + offset, nothing else
    i, j = torch.arange(Lp, device=dev)[:, None], torch.arange(Lp, device=dev)[None]
    col = (L - 1 + j - i + geo[0]).clamp(0, geo[1] - 1)
    inside = (valid[:, None, :, None] & valid[:, None, None, :]).expand(B, H, Lp, Lp)
    want = torch.zeros_like(band.transpose(0, 1)).scatter_add(3, col.expand(B, H, Lp, Lp), ds * inside)
    assert torch.equal(band.transpose(0, 1), want)


@gpu
@pytest.mark.parametrize("lens,H,D", [([1], 1, 64), ([63, 2], 3, 64), ([128, 1, 0, 64], 8, 128), ([500, 300, 411], 8, 64), ([70, 9], 3, 8), ([40, 33], 5, 24),
                                      ([100], 2, 96), ([300, 64], 4, 32)])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_att_pack_dqkv_leaves_the_column_sums(lens, H, D, accumulate):
    import ctypes
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import _lib

    pack = PackInfo(torch.tensor(lens, dtype=torch.int32), torch.device("cuda"))
    dev, bf, N, B, HD = "cuda", torch.bfloat16, pack.n, pack.batch, H * D
    Lp = (pack.max_len + 63) // 64 * 64
    torch.manual_seed(N)
    dqu, dqv, dk, dv = (torch.randn(B, Lp, HD, device=dev).to(bf) for _ in range(4))
    valid = torch.arange(Lp, device=dev)[None] < pack.lens[:, None]
    vp, i32 = ctypes.c_void_p, ctypes.c_int
    slices = _lib.bind("rb200_att_pack_slices", [i32, i32, i32])(N, H, D)
    got = torch.empty(N, 3 * HD, device=dev, dtype=bf)
    sq = torch.ones(3 * HD, device=dev)
    su = torch.ones(HD, device=dev) if accumulate else torch.full((slices, 2, HD), float("nan"), device=dev)
    sv = torch.ones(HD, device=dev)
    fn = _lib.bind("rb200_att_pack_dqkv", [vp] * 10 + [i32] * 5 + [vp])
    _lib.check(fn(dqu.data_ptr(), dqv.data_ptr(), dk.data_ptr(), dv.data_ptr(), pack.row_batch.data_ptr(), pack.row_pos.data_ptr(), got.data_ptr(),
                  sq.data_ptr(), su.data_ptr(), sv.data_ptr(), N, H, D, Lp, accumulate, _lib.stream_ptr()), "att_pack_dqkv")
    u, v, k, w = (t[valid].view(N, H, D) for t in (dqu, dqv, dk, dv))
    want = torch.stack([(u.float() + v.float()).to(bf), k, w], 2).reshape(N, 3 * HD)
    assert torch.equal(got, want)
    if not accumulate:
        assert (sq == 1).all() and (sv == 1).all()
        su, sv = su.sum(0) + 1
    else:
        assert ((sq.double() - 1 - want.double().sum(0)).abs() <= 1e-6 * want.double().abs().sum(0) + 1e-6).all()
    for s, t in ((su, u), (sv, v)):
        t = t.reshape(N, HD).double()
        assert ((s.double() - 1 - t.sum(0)).abs() <= 1e-6 * t.abs().sum(0) + 1e-6).all()


@gpu
@pytest.mark.parametrize("lens,H,slices", [([1], 1, 1), ([64, 65, 0, 128], 2, 4), ([320, 7, 201], 3, 5), ([384, 384], 1, 3), ([512, 1, 1, 511], 2, 1)])
def test_rel_flash_dpos_leaves_out_empty_blocks(lens, H, slices):
    """the position gradient against the whole product over a band that is zero outside the windows"""
    import ctypes
    from returnn_b200.ops import _lib, gemm as G

    dev, bf, HD, B, L = "cuda", torch.bfloat16, H * 64, len(lens), max(lens)
    Lp = (L + 63) // 64 * 64
    vp, i32, f32 = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
    geo = (ctypes.c_int * 2)()
    _lib.check(_lib.bind("rb200_rel_flash_band", [i32, i32, vp, vp])(Lp, L - 1, ctypes.addressof(geo), ctypes.addressof(geo) + 4), "band")
    off, width = geo[0], geo[1]
    torch.manual_seed(L)
    lens_t = torch.tensor(lens, dtype=torch.int32, device=dev)
    i, x = torch.arange(Lp, device=dev)[:, None], torch.arange(width, device=dev)[None]
    n = lens_t[:, None, None].long()
    window = (i < n) & (x >= L - 1 + off - i) & (x < L - 1 + off - i + n)
    band = (torch.randn(H, B, Lp, width, device=dev) * window).to(bf)
    qv = torch.randn(B, Lp, HD, device=dev).to(bf)
    part = torch.full((slices, width, HD), float("nan"), device=dev, dtype=torch.float32 if slices > 1 else bf)
    st = G.status_tensor(lens_t.device)
    fn = _lib.bind("rb200_rel_flash_dpos", [vp, vp, vp, vp, i32, i32, i32, i32, f32, i32, vp, vp])
    _lib.check(fn(band.data_ptr(), qv.data_ptr(), part.data_ptr(), lens_t.data_ptr(), B, H, Lp, L - 1, 0.125, slices, st.data_ptr(), _lib.stream_ptr()), "dpos")
    G.check_status()
    want = torch.einsum("hrx,rhd->xhd", band.double().view(H, B * Lp, width), qv.double().view(B * Lp, H, 64)).reshape(width, HD) * 0.125
    got = part.double().sum(0)
    # fp32 sums, one slice: the result in bf16
    assert (got - want).norm() <= (1e-5 if slices > 1 else 2 ** -8) * want.norm() + 1e-6
