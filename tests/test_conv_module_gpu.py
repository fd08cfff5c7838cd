"""
Fused conv-module kernels (GLU + depthwise conv + masked BatchNorm + SiLU on packed rows) against the torch math in fp32.
"""

import pytest
import torch

gpu = pytest.mark.gpu


class _BN:
    """the attributes of rf.BatchNorm that the op reads"""

    def __init__(self, C, device):
        class P:
            def __init__(self, t):
                self.raw_tensor = t

        self.affine = True
        self.eps = 1e-3
        self.momentum = 0.1
        self.gamma = P((torch.rand(C, device=device) + 0.5).requires_grad_(True))
        self.beta = P((torch.randn(C, device=device) * 0.1).requires_grad_(True))
        self.running_mean = P(torch.zeros(C, device=device))
        self.running_variance = P(torch.ones(C, device=device))


@gpu
@pytest.mark.parametrize("lens,C,K", [([50, 7, 33], 64, 32), ([334, 100, 1, 64, 200], 512, 32), ([40, 41], 128, 31), ([10], 64, 3)])
def test_conv_module_fwd_bwd(lens, C, K):
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import conv_module as cm, conv_module_native as cn, _lib

    torch.manual_seed(0)
    pack = PackInfo(torch.tensor(lens, dtype=torch.int32), torch.device("cuda"))
    N = pack.n
    assert cn.supports(C, K)
    x = torch.randn(N, 2 * C, device="cuda").to(torch.bfloat16).requires_grad_(True)
    filt = (torch.randn(C, 1, K, device="cuda") * 0.2).requires_grad_(True)
    bias = (torch.randn(C, device="cuda") * 0.1).requires_grad_(True)
    bn = _BN(C, "cuda")
    dz = torch.randn(N, C, device="cuda").to(torch.bfloat16)
    n0 = _lib.launch_count()
    z = cm.glu_dwconv_bn_silu(x, filt, bias, bn, pack, training=True)
    assert _lib.launch_count() > n0, "native kernels did not run"
    z.backward(dz)
    got = [z.float(), x.grad.float(), filt.grad.clone(), bias.grad.clone(), bn.gamma.raw_tensor.grad.clone(), bn.beta.raw_tensor.grad.clone()]
    rm_native = bn.running_mean.raw_tensor.clone()
    # reference: same function with the native path disabled, in fp32
    import os

    x32 = x.detach().float().requires_grad_(True)
    f32 = filt.detach().clone().requires_grad_(True)
    b32 = bias.detach().clone().requires_grad_(True)
    bn2 = _BN(C, "cuda")
    bn2.gamma.raw_tensor = bn.gamma.raw_tensor.detach().clone().requires_grad_(True)
    bn2.beta.raw_tensor = bn.beta.raw_tensor.detach().clone().requires_grad_(True)
    os.environ["RETURNN_B200_DISABLE_NATIVE"] = "1"
    try:
        orig = cn.available
        cn.available = lambda t: False
        zr = cm.glu_dwconv_bn_silu(x32, f32, b32, bn2, pack, training=True)
    finally:
        cn.available = orig
        del os.environ["RETURNN_B200_DISABLE_NATIVE"]
    zr.backward(dz.float())
    ref = [zr, x32.grad, f32.grad, b32.grad, bn2.gamma.raw_tensor.grad, bn2.beta.raw_tensor.grad]
    names = ["z", "dx", "dfilt", "dbias", "dgamma", "dbeta"]
    scale = max(1.0, N ** 0.5)
    tols = [0.05, 0.08, 0.05 * scale, 0.05 * scale, 0.05 * scale, 0.05 * scale]
    for n, g, r, t in zip(names, got, ref, tols):
        torch.testing.assert_close(g, r.float(), atol=t, rtol=5e-2, msg=lambda s, n=n: "%s: %s" % (n, s))
    torch.testing.assert_close(rm_native, bn2.running_mean.raw_tensor, atol=1e-2, rtol=1e-2)


@gpu
@pytest.mark.parametrize("lens,C,K", [
    ([1], 64, 32), ([31, 1, 32, 33, 0, 64], 64, 32), ([3] * 150, 128, 31), ([2000, 5], 64, 17), ([20] * 40 + [600], 256, 16), ([65, 7, 64], 512, 7),
    ([333, 100, 200, 40], 1024, 2), ([1] * 70, 64, 15), ([90, 120], 64, 33)])
@pytest.mark.parametrize("training", [True, False])
def test_conv_module_windows_against_float64(lens, C, K, training):
    """
    pieces and steps of the sliding-window kernels: short and empty sequences, pieces of one step and of many, both tap counts, and the old
    kernel beyond 32 taps. bf16 rounds the convolution, its gradient and the results once each: 2^-9 apiece, twice that in the sums over them
    """
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import conv_module as cm

    gen = torch.Generator("cuda").manual_seed(sum(lens) + K)
    pack = PackInfo(torch.tensor(lens, dtype=torch.int32), torch.device("cuda"))
    n = pack.n
    x = torch.randn(n, 2 * C, device="cuda", generator=gen).bfloat16().requires_grad_(True)
    filt = (torch.randn(C, 1, K, device="cuda", generator=gen) * K ** -0.5).requires_grad_(True)
    bias = (torch.randn(C, device="cuda", generator=gen) * 0.1).requires_grad_(not training)  # its gradient under batch statistics is 0
    bn = _BN(C, "cuda")
    dz = torch.randn(n, C, device="cuda", generator=gen).bfloat16()
    z = cm.glu_dwconv_bn_silu(x, filt, bias, bn, pack, training=training)
    leaves = [x, filt, bn.gamma.raw_tensor, bn.beta.raw_tensor] + ([] if training else [bias])
    got = [z, *torch.autograd.grad(z, leaves, dz)]
    x64, f64, g64, b64, c64 = (t.detach().double().requires_grad_(True) for t in (x, filt, bn.gamma.raw_tensor, bn.beta.raw_tensor, bias))
    h = x64[:, :C] * torch.sigmoid(x64[:, C:])
    ys, lo = [], 0
    for m in lens:
        if m:
            p = torch.nn.functional.pad(h[lo: lo + m].t()[None], ((K - 1) // 2, K - 1 - (K - 1) // 2))
            ys.append(torch.nn.functional.conv1d(p, f64, c64, groups=C)[0].t())
        lo += m
    y = torch.cat(ys)
    if training:
        y = (y - y.mean(0)) * torch.rsqrt(y.var(0, unbiased=False) + bn.eps)
    else:
        y = y * (1.0 + bn.eps) ** -0.5  # running statistics 0 and 1
    ref = torch.nn.functional.silu(y * g64 + b64)
    refs = [ref, *torch.autograd.grad(ref, [x64, f64, g64, b64] + ([] if training else [c64]), dz.double())]
    for name, a, b in zip(["z", "dx", "dfilt", "dgamma", "dbeta", "dbias"], got, refs):
        a = a.detach()
        if training and n == 1 and name not in ("z", "dbeta"):
            assert bool(torch.isfinite(a).all()), name  # the one row is its own mean: 0 but for the rounding of ds
            continue
        assert float((a.double() - b).norm()) <= 8e-3 * float(b.norm()), (name, float((a.double() - b).norm() / b.norm()))


@gpu
def test_conv_module_sequences_do_not_see_each_other():
    """not even through the zeros that fill up the taps: a NaN stays in its sequence"""
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import conv_module as cm

    lens, C = [40, 3, 70], 64
    pack = PackInfo(torch.tensor(lens, dtype=torch.int32), torch.device("cuda"))
    for K in (2, 7, 16, 31):
        x = torch.randn(sum(lens), 2 * C, device="cuda").bfloat16()
        x[41] = float("nan")
        x.requires_grad_(True)
        filt = torch.randn(C, 1, K, device="cuda")
        z = cm.glu_dwconv_bn_silu(x, filt, None, _BN(C, "cuda"), pack, training=False)
        (dx,) = torch.autograd.grad(z, [x], torch.ones_like(z))
        for t in (z, dx):
            assert bool(torch.isfinite(t[:40]).all()) and bool(torch.isfinite(t[43:]).all())


@gpu
@pytest.mark.parametrize("lens", [[1] + [0] * 70, [5, 3] + [0] * 300, [0] * 200 + [40], [0] * 70 + [30] + [0] * 70 + [300], [2, 1, 5]])
@pytest.mark.parametrize("C,K", [(64, 7), (512, 32)])
def test_conv_module_backward_with_many_empty_sequences(lens, C, K):
    """
    the zeros between the sequences make more pieces than there are partial sums in the scratch: nothing is written behind it, and the CTAs that
    take several pieces leave the sums of all. Sums of fp32 products in another order, dx rounded to bf16
    """
    import ctypes
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops import _lib

    gen = torch.Generator("cuda").manual_seed(len(lens) + K)
    pack = PackInfo(torch.tensor(lens, dtype=torch.int32), torch.device("cuda"))
    n = pack.n
    x = torch.randn(n, 2 * C, device="cuda", generator=gen).bfloat16()
    dy = torch.randn(n, C, device="cuda", generator=gen).bfloat16()
    filt = torch.randn(C, K, device="cuda", generator=gen) * K ** -0.5
    size = (n + 31) // 32 * C * (K + 1)
    part = torch.full((size + 64 * C * (K + 1),), 77.0, device="cuda")
    dx, dfilt, dbias = torch.empty_like(x), torch.empty_like(filt), torch.empty(C, device="cuda")
    vp, i32 = ctypes.c_void_p, ctypes.c_int
    fn = _lib.bind("rb200_glu_dwconv_bwd", [vp] * 10 + [i32] * 4 + [vp])
    _lib.check(fn(x.data_ptr(), dy.data_ptr(), filt.data_ptr(), pack.row_batch.data_ptr(), pack.row_pos.data_ptr(), pack.lens.data_ptr(), dx.data_ptr(),
                  part.data_ptr(), dfilt.data_ptr(), dbias.data_ptr(), n, pack.batch, C, K, _lib.stream_ptr()), "glu_dwconv_bwd")
    assert bool((part[size:] == 77.0).all())
    x64, f64 = x.double().requires_grad_(True), filt.double().requires_grad_(True)
    h = x64[:, :C] * torch.sigmoid(x64[:, C:])
    ys, lo = [], 0
    for m in lens:
        if m:
            p = torch.nn.functional.pad(h[lo: lo + m].t()[None], ((K - 1) // 2, K - 1 - (K - 1) // 2))
            ys.append(torch.nn.functional.conv1d(p, f64[:, None], groups=C)[0].t())
        lo += m
    want = torch.autograd.grad(torch.cat(ys), [x64, f64], dy.double())
    for a, b, tol in ((dx, want[0], 2 ** -8), (dfilt, want[1], 1e-5), (dbias, dy.double().sum(0), 1e-5)):
        assert float((a.double() - b).norm()) <= tol * float(b.norm()) + 1e-6
