"""Forward pass of the cross entropy on both sides of the rules that choose its form by classes, rows and type, against 64 bits."""

import pytest
import torch

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,v", [(3, 2), (1300, 1000), (5, 16383), (1184, 16384), (1185, 16391), (40, 4097), (7, 32000), (9, 4095), (3, 4096), (3, 4352), (3, 4353), (5, 8999), (5, 9000),
                                    (3, 12288), (3, 12289)])
@pytest.mark.parametrize("smoothing,arg", [(0.1, False), (0.0, True)])
def test_softmax_ce_forward(dtype, rows, v, smoothing, arg):
    import ctypes
    from returnn_b200.ops import _lib

    torch.manual_seed(rows + v)
    x = (torch.randn(rows, v, device="cuda") * 3).to(dtype)
    x[0] = torch.finfo(dtype).min if arg else x[0]
    x[-1, v // 2] = 60.0
    t = torch.randint(0, v, (rows,), device="cuda", dtype=torch.int32)
    loss, lse = torch.empty(2, rows, device="cuda")
    am = torch.full((rows,), -1, device="cuda", dtype=torch.int32)
    vp, i32, f32, i64 = ctypes.c_void_p, ctypes.c_int, ctypes.c_float, ctypes.c_longlong
    fn = _lib.bind("rb200_softmax_ce_fwd", [vp, vp, vp, vp, i64, i32, f32, i32, i32, vp, vp])
    _lib.check(fn(x.data_ptr(), t.data_ptr(), loss.data_ptr(), lse.data_ptr(), rows, v, smoothing, 1 if dtype == torch.bfloat16 else 0, 0,
                  am.data_ptr() if arg else None, _lib.stream_ptr()), "softmax_ce_fwd")
    d = x.double()
    want = torch.logsumexp(d, 1)
    pick = d.gather(1, t.long()[:, None])[:, 0]
    other = (v * want - d.sum(1) - (want - pick)) / (v - 1)
    ref = (1 - smoothing) * (want - pick) + smoothing * other
    ok = slice(1, None) if arg else slice(None)  # (row 0 of lowest values: the lse is their size, the loss log v in their rounding)
    # sums of v terms in fp32, an exponential of 2 ulp of an argument that is rounded to 2^-23 of at most 64
    assert ((lse[ok].double() - want[ok]).abs() <= 2.0**-16).all()
    assert ((loss[ok].double() - ref[ok]).abs() <= 2.0**-15 + 2.0**-20 * d[ok].abs().sum(1) / v).all()
    if arg:
        assert torch.isfinite(lse).all() and torch.equal(am.long(), x.float().argmax(1))


@gpu
@pytest.mark.parametrize("dtype,rows,v", [(torch.bfloat16, 1185, 28400), (torch.bfloat16, 1184, 28400), (torch.bfloat16, 1300, 1000), (torch.float32, 1185, 14200)])
def test_softmax_ce_gradient_by_order_of_rows(dtype, rows, v):
    """more rows than are resident at once and 64 MB of logits: last rows first; each row's gradient is that of its own target and factor"""
    from returnn_b200.ops.softmax_ce import softmax_cross_entropy

    g = torch.Generator(device="cuda").manual_seed(rows + v)
    x = (torch.randn(rows, v, generator=g, device="cuda") * 3).to(dtype).requires_grad_(True)
    t = torch.randint(0, v, (rows,), generator=g, device="cuda", dtype=torch.int32)
    f = torch.randn(rows, generator=g, device="cuda")
    (dx,) = torch.autograd.grad(softmax_cross_entropy(x, t), [x], f)
    at = [0, 1, rows // 2, rows - 2, rows - 1]
    want = torch.softmax(x[at].detach().double(), 1)
    want[torch.arange(len(at)), t[at].long()] -= 1.0
    want *= f[at].double()[:, None]
    # a rounding to the type and an exponential of 2 ulp of an argument that is rounded to 2^-20
    assert ((dx[at].double() - want).norm(dim=1) <= (2.0**-8 if dtype == torch.bfloat16 else 2.0**-17) * want.norm(dim=1)).all()
