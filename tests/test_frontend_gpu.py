"""Implicit-GEMM conv subsampling frontend against the torch (cuDNN / fp32) path: packed outputs and all parameter gradients."""

import pytest
import torch

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("lens", [[100, 57, 98, 3], [301, 300, 299]])
def test_frontend_native_matches_torch_path(lens):
    from returnn_b200.tensor import Dim
    from returnn_b200.frontend.encoder.conformer import ConformerEncoder, ConformerConvSubsample
    from returnn_b200.torch.frontend.bridge import rf_module_to_pt_module
    from returnn_b200.models import conformer_fused
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.utils.basic import BehaviorVersion

    BehaviorVersion._reset(24)
    torch.manual_seed(0)
    f = Dim(80, name="feat")
    enc = ConformerEncoder(f, Dim(64, name="model"), num_layers=1, num_heads=1, ff_dim=Dim(64, name="ff"), conv_kernel_size=3, dropout=0.0, att_dropout=0.0,
                           input_layer=ConformerConvSubsample(f, out_dims=[Dim(32, name="c1"), Dim(64, name="c2"), Dim(64, name="c3")],
                                                              filter_sizes=[(3, 3), (3, 3), (3, 3)], pool_sizes=[(1, 2)], strides=[(1, 1), (3, 1), (2, 1)]))
    pt = rf_module_to_pt_module(enc).to("cuda")
    with torch.no_grad():
        for n, p in pt.named_parameters():
            if "input_layer" in n and p.dim() == 1:
                p.normal_(0.0, 0.2)
    lens_host = torch.tensor(lens, dtype=torch.int32)
    feats = torch.randn(len(lens), max(lens), 80, device="cuda")
    params = [p for n, p in pt.named_parameters() if "input_layer" in n]
    # native
    x, pack = conformer_fused._frontend_native(enc, feats, lens_host)
    assert x is not None
    wgt = torch.randn_like(x.float())
    (x.float() * wgt).sum().backward()
    g_native = [p.grad.clone() for p in params]
    for p in params:
        p.grad = None
    # torch path in fp32
    W = conformer_fused._Weights(torch.float32)
    x_pad, lens2 = conformer_fused.frontend_subsample(enc, feats, lens_host, W)
    pack2 = PackInfo(lens2, feats.device, padded_len=x_pad.shape[1])
    ref = pack2.pack(x_pad)
    assert ref.shape == x.shape and pack2.lens_host.tolist() == pack.lens_host.tolist()
    (ref * wgt).sum().backward()
    torch.testing.assert_close(x.float(), ref, atol=0.06, rtol=0.05)
    errs = {}
    for p, g, (n, _) in zip(params, g_native, [(n, p) for n, p in pt.named_parameters() if "input_layer" in n]):
        scale = float(p.grad.abs().max()) + 1e-6
        errs[n] = (float((g.float() - p.grad).abs().max()) / scale, float(torch.nn.functional.cosine_similarity(g.float().flatten(), p.grad.flatten(), dim=0)))
    # bf16 activations and gradients through three layers against an fp32 reference: direction must agree closely, magnitudes within 10 %
    assert all(e < 0.1 and c > 0.995 for e, c in errs.values()), errs


@gpu
@pytest.mark.parametrize("lens,F,C", [([1], 2, 8), ([7, 8, 9, 0], 6, 32), ([17, 3], 80, 64), ([40, 33], 4, 256)])
@pytest.mark.parametrize("with_bias", [True, False])
def test_conv1_relu_pool_backward(lens, F, C, with_bias):
    """filter and bias gradient of convolution, ReLU and pooling over two features against 64 bits: lengths around the runs of 8 frames"""
    import ctypes
    from returnn_b200.ops import _lib

    torch.manual_seed(F + C)
    dev, bf, B, T = "cuda", torch.bfloat16, len(lens), max(lens)
    x = torch.randn(B, T, F, device=dev).to(bf)
    w, b = torch.randn(C, 1, 3, 3, device=dev), torch.randn(C, device=dev) * 0.3
    dy = torch.randn(B, T, F // 2, C, device=dev).to(bf)
    n = torch.tensor(lens, dtype=torch.int32, device=dev)
    dw, db = torch.ones(C, 9, device=dev), torch.ones(C, device=dev)
    vp, i32 = ctypes.c_void_p, ctypes.c_int
    fn = _lib.bind("rb200_conv1_relu_pool_bwd", [vp, vp, vp, vp, vp, i32, i32, i32, i32, vp, vp, vp])
    _lib.check(fn(x.data_ptr(), w.data_ptr(), b.data_ptr() if with_bias else None, n.data_ptr(), dy.data_ptr(), B, T, F, C, dw.data_ptr(), db.data_ptr(),
                  _lib.stream_ptr()), "conv1_relu_pool_bwd")
    valid = (torch.arange(T, device=dev)[None] < n[:, None]).double()
    w64, b64 = w.double().requires_grad_(True), (b if with_bias else b * 0).double().requires_grad_(True)
    y = torch.nn.functional.conv2d(x.double()[:, None] * valid[:, None, :, None], w64, b64, padding=1)
    y = torch.nn.functional.max_pool2d(torch.relu(y), (1, 2)).permute(0, 2, 3, 1)
    (y * dy.double() * valid[:, :, None, None]).sum().backward()
    # 32-bit sums of at most 3000 products; inputs drawn from a continuous distribution: no ties of the two candidates but by chance
    for got, want in ((dw - 1, w64.grad.view(C, 9)), (db - 1, b64.grad)):
        assert (got.double() - want).norm() <= 1e-3 * want.norm() + 1e-5


@gpu
def test_frontend_lengths_beyond_the_batch_read_no_frames_behind_it():
    """rows and parameter gradients as with the batch's own length, for the output frames that do not see its end"""
    from returnn_b200.tensor import Dim
    from returnn_b200.frontend.encoder.conformer import ConformerEncoder, ConformerConvSubsample
    from returnn_b200.torch.frontend.bridge import rf_module_to_pt_module
    from returnn_b200.models import conformer_fused
    from returnn_b200.utils.basic import BehaviorVersion

    BehaviorVersion._reset(24)
    torch.manual_seed(0)
    f = Dim(80, name="feat")
    enc = ConformerEncoder(f, Dim(64, name="model"), num_layers=1, num_heads=1, ff_dim=Dim(64, name="ff"), conv_kernel_size=3, dropout=0.0, att_dropout=0.0,
                           input_layer=ConformerConvSubsample(f, out_dims=[Dim(32, name="c1"), Dim(64, name="c2"), Dim(64, name="c3")],
                                                              filter_sizes=[(3, 3), (3, 3), (3, 3)], pool_sizes=[(1, 2)], strides=[(1, 1), (3, 1), (2, 1)]))
    pt = rf_module_to_pt_module(enc).to("cuda")
    params = [p for n, p in pt.named_parameters() if "input_layer" in n]
    T = 120
    feats = torch.randn(2, T, 80, device="cuda")
    wgt = torch.randn(2, T // 6 - 2, 1, device="cuda")
    res = []
    for n in (T, T + 11):
        x, pack = conformer_fused._frontend_native(enc, feats, torch.tensor([n, n], dtype=torch.int32))
        rows = x[: pack.n].view(2, -1, x.shape[1])[:, : T // 6 - 2]
        grads = torch.autograd.grad((rows.float() * wgt).sum(), params, allow_unused=True)
        res.append((rows.detach(), [g for g in grads if g is not None]))
    assert float((res[0][0].float() - res[1][0].float()).norm()) <= 1e-3 * float(res[0][0].float().norm()) and len(res[0][1]) >= 6
    for a, b in zip(res[0][1], res[1][1]):  # 32-bit sums in another order
        assert float((a - b).norm()) <= 1e-3 * float(a.norm())
