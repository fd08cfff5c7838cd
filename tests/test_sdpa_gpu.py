"""scaled-dot-product attention kernels against plain PyTorch fp32"""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(B, H, D, Tq, Tk, causal, with_lens, seed=0):
    from returnn_b200.ops import sdpa as S

    torch.manual_seed(seed)
    dev = torch.device("cuda")
    bf = torch.bfloat16
    q = (torch.randn(B, Tq, H * D, device=dev) * 0.7).to(bf).requires_grad_(True)
    k = (torch.randn(B, Tk, H * D, device=dev) * 0.7).to(bf).requires_grad_(True)
    v = (torch.randn(B, Tk, H * D, device=dev) * 0.7).to(bf).requires_grad_(True)
    lens = torch.randint(max(1, Tk // 2), Tk + 1, (B,), device=dev, dtype=torch.int32) if with_lens else None
    assert S.supports(q, k, H)
    out = S.sdpa(q, k, v, num_heads=H, k_lens=lens, causal=causal)
    w = torch.randn_like(out, dtype=torch.float32)
    (out.float() * w).sum().backward()
    qr, kr, vr = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    ref = S.sdpa_reference(qr, kr, vr, num_heads=H, k_lens=lens, causal=causal)
    (ref * w).sum().backward()
    torch.testing.assert_close(out.float(), ref, atol=2e-2, rtol=2e-2)
    for got, want, name in ((q.grad, qr.grad, "dq"), (k.grad, kr.grad, "dk"), (v.grad, vr.grad, "dv")):
        err = (got.float() - want).abs().max().item()
        scale = want.abs().max().item() + 1e-6
        assert err / scale < 3e-2, (name, err, scale)


@pytest.mark.parametrize("B,H,D,Tq,Tk,causal,with_lens", [
    (3, 2, 64, 70, 70, False, True),     # encoder self attention with padding
    (2, 4, 64, 33, 33, True, False),     # causal decoder self attention
    (2, 2, 64, 17, 130, False, True),    # cross attention: short queries, long padded keys
    (1, 1, 128, 1, 65, True, False),     # one decoding step against a cache (the query is the last position)
    (2, 8, 64, 128, 192, False, False),  # sizes on tile boundaries
    (2, 2, 64, 40, 300, False, True),    # several tiles of keys
    (1, 2, 64, 64, 600, False, True),
    (2, 2, 64, 200, 200, True, True),    # causal with padding
])
def test_sdpa_matches_reference(B, H, D, Tq, Tk, causal, with_lens):
    _case(B, H, D, Tq, Tk, causal, with_lens)


@pytest.mark.parametrize("B,H,D,Tq,Tk,causal,with_lens", [
    (2, 2, 128, 30, 50, False, True),    # the softmax kernels between two products: eight lanes per row of keys
    (2, 1, 128, 70, 100, False, True),   # sixteen
    (2, 2, 128, 200, 200, True, True),   # causal with padding, a whole warp per row
    (2, 2, 128, 40, 300, False, True),   # rows of two register chunks per lane
    (1, 2, 192, 64, 600, False, True),   # ... and of four
    (1, 1, 128, 33, 1100, True, True),   # scores in 32 bits
])
def test_sdpa_matches_reference_for_other_head_dims(B, H, D, Tq, Tk, causal, with_lens):
    _case(B, H, D, Tq, Tk, causal, with_lens)


def test_sdpa_dropout_statistics_and_4d_entry():
    from returnn_b200.ops import sdpa as S, attention as A

    torch.manual_seed(1)
    dev = torch.device("cuda")
    B, H, D, T = 2, 2, 64, 96
    q = torch.randn(B, T, H * D, device=dev).to(torch.bfloat16)
    k = torch.randn(B, T, H * D, device=dev).to(torch.bfloat16)
    v = torch.ones(B, T, H * D, device=dev).to(torch.bfloat16)
    # with constant values the output is the kept probability mass / (1-p): mean 1, and not identically 1
    out = S.sdpa(q, k, v, num_heads=H, dropout_p=0.5).float()
    assert abs(out.mean().item() - 1.0) < 0.05 and out.std().item() > 0.01
    # the [B, H, T, D] entry used by rf.dot_attention
    q4 = q.view(B, T, H, D).transpose(1, 2)
    k4 = k.view(B, T, H, D).transpose(1, 2)
    vv = torch.randn(B, T, H * D, device=dev).to(torch.bfloat16)
    v4 = vv.view(B, T, H, D).transpose(1, 2)
    lens = torch.tensor([96, 50], device=dev, dtype=torch.int32)
    got = A.sdpa(q4, k4, v4, kv_lens=lens, scale=D ** -0.5, causal=False)
    want = A.sdpa_reference(q4.float(), k4.float(), v4.float(), kv_lens=lens, scale=D ** -0.5, causal=False)
    torch.testing.assert_close(got.float(), want, atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("layout", ["per_head_interleaved", "three_blocks"])
def test_sdpa_heads_reads_slices_of_a_fused_projection_in_place(layout):
    """q / k / v as strided views of one [B, T, 3 * H * D] tensor (both common column orders): same result and gradients as on copies"""
    from returnn_b200.ops import sdpa as S

    torch.manual_seed(3)
    dev = torch.device("cuda")
    B, T, H, D = 3, 75, 4, 64
    qkv = (torch.randn(B, T, 3 * H * D, device=dev) * 0.7).to(torch.bfloat16).requires_grad_(True)
    lens = torch.tensor([75, 40, 9], device=dev, dtype=torch.int32)

    def split(x):
        if layout == "per_head_interleaved":  # [.., H, 3 * D] -> three [.., H, D] slices
            x4 = x.view(B, T, H, 3 * D)
            return x4[..., :D], x4[..., D: 2 * D], x4[..., 2 * D:]
        x4 = x.view(B, T, 3, H, D)
        return x4[:, :, 0], x4[:, :, 1], x4[:, :, 2]

    q, k, v = split(qkv)
    assert not q.is_contiguous() and S._rows(q)[0].data_ptr() == q.data_ptr()  # addressed in place
    w = torch.randn(B, T, H, D, device=dev)
    out = S.sdpa_heads(q, k, v, k_lens=lens)
    (out.float() * w).sum().backward()
    got = qkv.grad.clone()
    qkv.grad = None
    qc, kc, vc = (t.contiguous().view(B, T, H * D) for t in split(qkv))
    ref = S.sdpa_reference(qc, kc, vc, num_heads=H, k_lens=lens).view(B, T, H, D)
    (ref * w).sum().backward()
    torch.testing.assert_close(out.float(), ref, atol=2e-2, rtol=2e-2)
    scale = float(qkv.grad.abs().max())
    assert float((got.float() - qkv.grad.float()).abs().max()) / scale < 3e-2


@pytest.mark.parametrize("Tq,Tk,causal,with_lens", [
    (1, 1, False, False),       # one score
    (63, 65, False, True),      # a key into the second tile of 64
    (65, 64, False, False),
    (128, 128, True, False),    # whole tiles
    (129, 257, True, True),     # one row into the second tile of queries; causal with more keys than queries
    (200, 70, True, False),     # more queries than keys: the first queries see no key and get zeros
])
def test_sdpa_head_dim_64_tile_edges(Tq, Tk, causal, with_lens):
    _case(2, 3, 64, Tq, Tk, causal, with_lens, seed=Tq)


@pytest.mark.parametrize("T", [64, 50])
def test_sdpa_head_dim_64_dropout_gradients(T):
    """with the identity as values the output is the dropped probabilities: they give the mask, which the backward pass has to use as well"""
    from returnn_b200.ops import sdpa as S
    from returnn_b200.ops.elementwise import _seed_tensor

    torch.manual_seed(5)
    dev, B, H, D, p = torch.device("cuda"), 2, 2, 64, 0.3
    q, k, v = ((torch.randn(B, T, H, D, device=dev) * 0.7).to(torch.bfloat16).requires_grad_(True) for _ in range(3))
    eye = torch.eye(T, D, device=dev, dtype=torch.bfloat16)[None, :, None].expand(B, T, H, D).contiguous()
    seed = _seed_tensor(q.device)
    state = seed.clone()
    probs = S.sdpa_heads(q, k, eye, dropout_p=p)
    mask = (probs.detach().float()[..., :T] > 0).transpose(1, 2).float()  # [B, H, T, T]
    assert abs(mask.mean().item() - (1 - p)) < 0.03
    seed.copy_(state)
    out = S.sdpa_heads(q, k, v, dropout_p=p)
    w = torch.randn_like(out, dtype=torch.float32)
    (out.float() * w).sum().backward()
    qr, kr, vr = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    att = torch.softmax(torch.einsum("bihd,bjhd->bhij", qr, kr) * D ** -0.5, -1) * mask / (1 - p)
    ref = torch.einsum("bhij,bjhd->bihd", att, vr)
    (ref * w).sum().backward()
    torch.testing.assert_close(out.float(), ref, atol=2e-2, rtol=2e-2)
    for got, want in ((q.grad, qr.grad), (k.grad, kr.grad), (v.grad, vr.grad)):
        assert (got.float() - want).norm() / want.norm() < 1e-2  # bf16 probabilities and results: 2^-9 each per element


@pytest.mark.parametrize("D", [64, 128])
def test_sdpa_without_keys_or_queries_is_refused(D):
    """no keys: nothing to attend to; no queries: no gradient of the keys. Both are errors for every head dim, not results without values"""
    from returnn_b200.ops import sdpa as S

    q, none = torch.zeros(2, 3, 2, D, device="cuda", dtype=torch.bfloat16), torch.zeros(2, 0, 2, D, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(RuntimeError):
        S.sdpa_heads(q, none, none)
    k, v = q.clone().requires_grad_(True), q.clone().requires_grad_(True)
    out = S.sdpa_heads(none, k, v)
    assert out.shape == (2, 0, 2, D)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(out, [k, v], out.detach())


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("p", [1.0, 1.5])
def test_sdpa_dropout_rate_of_one_or_more_is_refused(D, p):
    from returnn_b200.ops import sdpa as S

    q = torch.zeros(1, 3, 2, D, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(RuntimeError):
        S.sdpa_heads(q, q, q, dropout_p=p)


def test_sdpa_dropout_streams_of_the_two_forms_are_apart():
    """
    the fused kernels (head dim 64) count in scores and the softmax kernels (128) in groups of four: if both drew from one stream, group c of
    the latter would repeat the decisions of the former at score c. With the identity as values the outputs show the decisions.
    """
    from returnn_b200.ops import sdpa as S
    from returnn_b200.ops.elementwise import _seed_tensor

    dev, p, kept = torch.zeros(1, device="cuda").device, 0.3, {}
    seed = _seed_tensor(dev)
    for T in (64, 128):
        seed[1] = 0  # the same position of the generator for both
        zero = torch.zeros(1, T, 1, T, device=dev, dtype=torch.bfloat16)
        eye = torch.eye(T, device=dev, dtype=torch.bfloat16)[None, :, None]
        kept[T] = (S.sdpa_heads(zero, zero, eye, dropout_p=p)[0, :, 0] > 0).view(-1, 4)
    n = 64 * 64 // 4
    same = (kept[64][:n] == kept[128][torch.arange(n, device=dev) * 4]).float().mean().item()
    # independent decisions agree with probability p^2 + (1-p)^2 = 0.58; 4096 of them scatter by 0.008
    assert abs(same - (p * p + (1 - p) * (1 - p))) < 0.04


def test_sdpa_result_of_the_fused_kernels_may_be_changed_in_place():
    from returnn_b200.ops import sdpa as S

    torch.manual_seed(4)
    D = 64
    q, k, v = (torch.randn(2, 70, 2, D, device="cuda", dtype=torch.bfloat16).requires_grad_(True) for _ in range(3))
    w = torch.randn(2, 70, 2, D, device="cuda", dtype=torch.bfloat16)
    want = torch.autograd.grad(S.sdpa_heads(q, k, v), [q, k, v], w * 2)
    out = S.sdpa_heads(q, k, v)
    out.mul_(2)
    for a, b in zip(torch.autograd.grad(out, [q, k, v], w), want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("T,causal", [(512, False), (300, True)])
def test_sdpa_query_gradient_where_values_share_an_offset(T, causal):
    """
    An offset common to all keys or all values leaves the query gradient as it is: the rows of dS sum to zero. That holds as far as the row
    sums of P * dP are known, here 24 |dO| = 24 * 8, where dS itself is 8 P. What remains is the 16-bit rounding of the n probabilities in
    the output, 24 * 8 * 0.0009 / sqrt(n) per row, times the common key 4, against 8 / sqrt(n): 0.09 for every n (row sums from the output
    in 16 bits: 24 * 8 * 0.0009 * 4 against 8 / sqrt(n), 2 at n = 512).
    """
    from returnn_b200.ops import sdpa as S

    torch.manual_seed(6)
    D = 64
    dev = torch.device("cuda")
    q = (torch.randn(1, T, 2, D, device=dev) * 0.02).to(torch.bfloat16)
    k = (torch.randn(1, T, 2, D, device=dev) + 4).to(torch.bfloat16)
    v = (torch.randn(1, T, 2, D, device=dev) + 24).to(torch.bfloat16)
    dy = torch.randn(1, T, 2, D, device=dev, dtype=torch.bfloat16)
    x = [t.clone().requires_grad_(True) for t in (q, k, v)]
    got = torch.autograd.grad(S.sdpa_heads(*x, causal=causal), x[:1], dy)[0]
    r = [t.double().requires_grad_(True) for t in (q, k, v)]
    want = torch.autograd.grad(S.sdpa_reference(*(t.flatten(2) for t in r), num_heads=2, causal=causal), r[:1], dy.float().flatten(2))[0]
    err = ((got.double() - want).norm() / want.norm()).item()
    assert err <= 0.2, err


@pytest.mark.parametrize("D,Tq,Tk,causal", [(64, 300, 300, True), (64, 150, 270, False), (64, 129, 200, True), (128, 140, 140, True), (128, 40, 300, False)])
def test_sdpa_dropout_gradients_over_several_tiles(D, Tq, Tk, causal):
    """the decisions of all tiles, read out block by block: with the identity on a block of keys as values the output is the kept probabilities"""
    from returnn_b200.ops import sdpa as S
    from returnn_b200.ops.elementwise import _seed_tensor

    torch.manual_seed(7)
    B, H, p = 2, 2, 0.2
    q, k, v = ((torch.randn(B, t, H, D, device="cuda") * 0.7).to(torch.bfloat16).requires_grad_(True) for t in (Tq, Tk, Tk))
    seed = _seed_tensor(q.device)
    state = seed.clone()
    mask = torch.zeros(B, H, Tq, Tk, device="cuda")
    for j in range(0, Tk, D):
        block = torch.zeros(B, Tk, H, D, device="cuda", dtype=torch.bfloat16)
        n = min(D, Tk - j)
        block[:, j: j + n, :, :n] = torch.eye(n, device="cuda", dtype=torch.bfloat16)[:, None]
        seed.copy_(state)
        mask[..., j: j + n] = (S.sdpa_heads(q.detach(), k.detach(), block, causal=causal, dropout_p=p)[..., :n] > 0).transpose(1, 2).float()
    seen = torch.ones(Tq, Tk, device="cuda").tril(Tk - Tq) if causal else torch.ones(Tq, Tk, device="cuda")
    assert abs((mask.sum() / (seen.sum() * B * H)).item() - (1 - p)) < 0.02
    seed.copy_(state)
    out = S.sdpa_heads(q, k, v, causal=causal, dropout_p=p)
    w = torch.randn_like(out)
    got = torch.autograd.grad(out, [q, k, v], w)
    r = [t.detach().double().requires_grad_(True) for t in (q, k, v)]
    s = (torch.einsum("bihd,bjhd->bhij", r[0], r[1]) * D ** -0.5).masked_fill(seen == 0, float("-inf"))
    ref = torch.einsum("bhij,bjhd->bihd", torch.softmax(s, -1) * mask / (1 - p), r[2])
    assert (out.double() - ref).norm() <= 1e-2 * ref.norm()
    for a, b in zip(got, torch.autograd.grad(ref, r, w.double())):
        # fused: probabilities, dS and results rounded to bf16, 2^-9 each; other head dims: scores and dP as well
        assert (a.double() - b).norm() <= (1e-2 if D == 64 else 2e-2) * b.norm()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_sdpa_sequence_without_visible_keys(D, causal):
    """a length of zero in the batch: zeros for its queries, no gradient into its keys and values, nothing of it in the other entries"""
    from returnn_b200.ops import sdpa as S

    torch.manual_seed(11)
    lens = torch.tensor([0, 70, 0], device="cuda", dtype=torch.int32)
    x = [torch.randn(3, 90, 2, D, device="cuda").to(torch.bfloat16).requires_grad_(True) for _ in range(3)]
    w = torch.randn(3, 90, 2, D, device="cuda").to(torch.bfloat16)
    out = S.sdpa_heads(*x, k_lens=lens, causal=causal)
    got = torch.autograd.grad(out, x, w)
    one = [t.detach()[1:2].clone().requires_grad_(True) for t in x]
    want_out = S.sdpa_heads(*one, k_lens=lens[1:2].clone(), causal=causal)
    want = torch.autograd.grad(want_out, one, w[1:2])
    for a, b in zip((out, *got), (want_out, *want)):
        assert torch.equal(a[1:2], b) and float(a[0].abs().max()) == 0.0 and float(a[2].abs().max()) == 0.0
