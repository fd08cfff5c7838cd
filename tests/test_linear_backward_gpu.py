"""Backward kernels of the linear layer at the edges of their forms: sliced weight gradients on CTA pairs, the wide form of the activation gradient,
epilogues of the pair kernel at ragged sizes, NaN through the exchanged matrices of the BLSTM."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n", [(600, 160, 136), (1100, 512, 520), (4097, 288, 264), (700, 144, 136), (512, 136, 2048)])
def test_weight_gradient_in_slices(m, k, n):
    """k = 160, 288, 512: slices on CTA pairs; 144 and 136 are no multiples of 32 rows: batched product"""
    from returnn_b200.ops import gemm as G, guard

    g = torch.Generator(device="cuda").manual_seed(m)
    x, dy = (torch.randn(m, c, generator=g, device="cuda").bfloat16() for c in (k, n))
    with guard.CanaryAllocations() as canary:
        dw, again = G._weight_grad(x, dy), G._weight_grad(x, dy)
    canary.check()
    G.check_status()
    ref = x.double().t() @ dy.double()
    assert torch.equal(dw, again)
    # 32-bit sums of m products of 16-bit values: sqrt(m) roundings of 2^-24 of sums of the size of the result, with room for the worst element
    assert float((dw - ref).abs().max()) <= 2 ** -24 * m ** 0.5 * 32 * float(ref.std())


@pytest.mark.parametrize("rows,cols,act", [(6000, 2056, "silu"), (12100, 1000, None), (46900, 256, "relu"), (1201, 10000, "gelu"), (5800, 2056, "silu"), (12000, 1536, None), (317, 37888, None),
                                           (317, 37896, None), (310, 40000, "relu"), (33, 47400, None), (4100, 1024, None), (3, 1032, None)])
def test_activation_gradient_and_column_sums(rows, cols, act):
    """wide form (ragged in rows and columns, at the ends of its range, more CTAs than are resident at once) and its neighbours in the narrow one"""
    from returnn_b200.ops import gemm as G

    g = torch.Generator(device="cuda").manual_seed(rows)
    z, dy = (torch.randn(rows, cols, generator=g, device="cuda").bfloat16() for _ in range(2))
    db = torch.full((cols,), float("nan"), device="cuda")
    dz = G._grad_pre(dy, z if act else None, act, db)
    ref = G._act_grad(z.double(), dy.double(), act) if act else dy.double()
    # one rounding to bf16 of a value that is within a few 2^-24 of the exact one
    assert float((dz.double() - ref).abs().max()) <= 2 ** -8 * float(ref.abs().max())
    assert float((dz.double() - ref).norm()) <= 2 ** -8 * float(ref.norm())
    torch.testing.assert_close(db.double(), dz.double().sum(0), rtol=0, atol=rows * 2 ** -24 * float(dz.abs().max()) * 8)


@pytest.mark.parametrize("m,n,k", [(129, 136, 64), (257, 264, 72), (300, 520, 512), (385, 1000, 200)])
@pytest.mark.parametrize("form", ["plain", "bias", "two", "resid", "dact", "f32", "drop_two", "drop_resid", "drop_dact", "odd"])
def test_pair_epilogues(m, n, k, form):
    """every form of the epilogue at ragged sizes; with dropout the mask is that of the stand-alone dropout kernel at the same counters"""
    from returnn_b200.ops import gemm as G
    from returnn_b200.ops.elementwise import dropout_with_state

    g = torch.Generator(device="cuda").manual_seed(m + n)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    if form == "odd":
        n -= 3
    a, b, z, r, bias = rnd(m, k), rnd(n, k), rnd(m, n), rnd(m, n), torch.randn(n, generator=g, device="cuda")
    out = torch.full((m + 1, n), 7.0, device="cuda", dtype=torch.float32 if form == "f32" else torch.bfloat16)
    kw = dict(m=m, n=n, k=k, a_mn_major=False, b_mn_major=False, out=out[:m])
    acc = a.double() @ b.double().t()
    second = torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
    drop = dict(dropout_p=0.25, dropout_seed=torch.tensor([5], device="cuda"), dropout_offset=torch.tensor([9], device="cuda")) if "drop" in form else {}
    mask = torch.ones(m, n, dtype=torch.double, device="cuda")
    if drop:
        ones = torch.ones(m, n, dtype=torch.bfloat16, device="cuda")
        mask = (dropout_with_state(ones, 0.25, drop["dropout_seed"], drop["dropout_offset"] + 1000) > 0).double()
        drop["dropout_site"] = 1000
    s = torch.sigmoid(z.double())
    if form in ("plain", "f32", "odd"):
        ref = acc
        G.gemm(a, b, **kw)
    elif form == "bias":
        ref = torch.relu(acc + bias)
        G.gemm(a, b, bias=bias, act="relu", **kw)
    elif "two" in form:
        ref = acc + bias
        G.gemm(a, b, bias=bias, act="silu", want_act_output=True, out_act=second, **drop, **kw)
    elif "resid" in form:
        ref = r.double() + 0.5 * (acc + bias) * mask / (0.75 if drop else 1.0)
        G.gemm(a, b, bias=bias, resid=r, res_scale=0.5, **drop, **kw)
    else:
        ref = acc * (s * (1 + z.double() * (1 - s))) * mask / (0.75 if drop else 1.0)
        G.gemm(a, b, dact_z=z, act="silu", **drop, **kw)
    G.check_status()
    assert float((out[m] - 7.0).abs().max()) == 0.0
    y = out[:m].double()
    # tanh.approx of the SiLU forms is within 2^-11 of its result, the rest is one rounding to bf16 (2^-9) of sums of 32 bits
    tol = 2 ** -20 if form == "f32" else 2 ** -8
    assert float((y - ref).norm()) <= tol * float(ref.norm())
    if form == "drop_dact":
        assert bool((y[mask == 0] == 0).all())
    if "two" in form:
        act = torch.nn.functional.silu(ref) * mask / (0.75 if drop else 1.0)
        assert float((second.double() - act).norm()) <= 2 ** -8 * float(act.norm())
        assert bool((second[mask == 0] == 0).all())


@pytest.mark.parametrize("m,n", [(6336, 6320), (6272, 6368)])
def test_adding_onto_a_matrix_beyond_the_cache(m, n):
    """40 M elements on: another epilogue"""
    from returnn_b200.ops import gemm as G

    g = torch.Generator(device="cuda").manual_seed(m)
    a, b = (torch.randn(r, 72, generator=g, device="cuda").bfloat16() for r in (m, n))
    out = torch.full((m, n), 2.0, device="cuda")
    G.gemm(a, b, m=m, n=n, k=72, a_mn_major=False, b_mn_major=False, out=out, atomic=True)
    G.check_status()
    # sums of 72 products and of the two terms in 32 bits: 2^-24 of values of up to 64 each
    assert float((out - 2.0 - a.float() @ b.float().t()).abs().max()) <= 72 * 2 ** -24 * 64


@pytest.mark.parametrize("rows", [3, 20])
def test_blstm_passes_nan_on_without_waiting(rows):
    """NaN in one sequence (every NaN that a conversion can give) stays there, and no wait runs out: what marks unwritten values is another one"""
    from returnn_b200.ops import gemm as G
    from returnn_b200.ops.lstm_native import blstm

    T, H, n_in = 6, 128, 16
    g = torch.Generator(device="cuda").manual_seed(rows)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda") * 0.3  # noqa: E731
    par = [tuple(rnd(*s) for s in ((4 * H, n_in), (4 * H, H), (4 * H,))) for _ in range(2)]
    zero = torch.zeros(rows, H, device="cuda")
    res = []
    for nan in (False, True):
        torch.manual_seed(0)
        x = torch.randn(T, rows, n_in, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").bfloat16()
        if nan:
            x.view(torch.int16)[2, 1] = -1  # the bits 0xffff
        x.requires_grad_(True)
        (yf, _, cf), (yb, _, cb) = blstm(x, None, par[0], par[1], zero, zero, zero, zero)
        (dx,) = torch.autograd.grad([yf, yb], [x], [torch.ones_like(yf), torch.ones_like(yb)])
        res.append((yf, yb, cf, cb, dx))
    G.check_status()
    others = [i for i in range(rows) if i != 1]
    for a, b in zip(*res):
        rest = (slice(None),) if a.dim() == 3 else ()
        assert torch.equal(a[rest + (others,)], b[rest + (others,)])
    assert bool(res[1][0][2:, 1].isnan().all()) and bool(res[1][1][:3, 1].isnan().all()) and bool(res[1][4][:, 1].isnan().all())
    assert not bool(res[1][0][:2, 1].isnan().any())
