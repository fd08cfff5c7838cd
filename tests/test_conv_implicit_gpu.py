"""3x3 convolutions without patch matrices (forward, data gradient, filter gradient) against fp32 convolutions of the same bf16 operands."""

import pytest
import torch

gpu = pytest.mark.gpu


def _conv_ref(x, w, stride, pad, To):
    """x [B, T, F, c], w [n, c, 3, 3] -> [B, To, F, n]"""
    right = max((To - 1) * stride + 3 - pad - x.shape[1], 0)
    y = torch.nn.functional.conv2d(torch.nn.functional.pad(x.permute(0, 3, 1, 2), (1, 1, pad, right)), w, stride=(stride, 1))
    return y[:, :, :To].permute(0, 2, 3, 1)


@gpu
@pytest.mark.parametrize("F,c,n", [(8, 32, 64), (40, 32, 64), (40, 64, 64), (80, 64, 64), (64, 64, 32), (24, 32, 32), (72, 32, 64)])
@pytest.mark.parametrize("stride,pad,lens,packed", [(3, 1, [50, 0, 31, 1], False), (2, 0, [50, 47, 3], True), (1, 1, [5, 17], True), (4, 2, [23, 40], False), (2, 1, [700, 411], False)])
def test_conv3x3(F, c, n, stride, pad, lens, packed):
    from returnn_b200.ops import frontend_native as fe

    assert fe._implicit(F, c, n)
    torch.backends.cudnn.allow_tf32 = False
    torch.manual_seed(F + c + n + stride)
    B, T = len(lens), max(lens) + 2  # (a padded length above the longest)
    To = -(-T // stride)
    dev, bf = "cuda", torch.bfloat16
    lens_in = torch.tensor(lens, dtype=torch.int32, device=dev)
    lens_out = (lens_in + stride - 1) // stride
    x = torch.randn(B, T, F, c, device=dev).to(bf)
    w = (torch.randn(n, c, 3, 3, device=dev) * 0.1).to(bf)
    bias = torch.randn(n, device=dev)
    live = (torch.arange(T, device=dev)[None] < lens_in[:, None])[:, :, None, None]
    live_out = (torch.arange(To, device=dev)[None] < lens_out[:, None])
    xm, wf = x.float() * live, w.float()
    row_batch = row_pos = cu = None
    n_frames = B * To
    pick = torch.ones_like(live_out)
    if packed:
        pick = live_out
        rows = live_out.nonzero()
        row_batch, row_pos, n_frames = rows[:, 0].int().contiguous(), rows[:, 1].int().contiguous(), rows.shape[0]
        cu = torch.cat([torch.zeros(1, dtype=torch.int32, device=dev), lens_out.cumsum(0).int()])
    # bf16 results: half a unit of 2^-8, and the order of 9 c products in fp32
    eps = 9 * c * 2.0**-24

    y = torch.full((n_frames, F, n), float("nan"), device=dev, dtype=bf)
    fe._conv(x, w.permute(0, 2, 3, 1).reshape(n, 9 * c).contiguous(), bias, None, y, lens_in, None, None, row_batch, row_pos, B, T, To, F, c, n, stride, pad,
             n_frames, False)
    ref = torch.relu(_conv_ref(xm, wf, stride, pad, To) + bias)[pick].view(n_frames, F, n)
    mag = _conv_ref(xm.abs(), wf.abs(), stride, pad, To)[pick].view(n_frames, F, n) + bias.abs()
    assert ((y.float() - ref).abs() <= 2.0**-8 * ref.abs() + eps * mag).all()

    dy = torch.randn(n_frames, F, n, device=dev).to(bf)
    full = torch.zeros(B, To, F, n, device=dev)
    full[pick] = dy.float().view(-1, F, n)
    full = full * live_out[:, :, None, None]  # frames past a sequence's output length give nothing to the data gradient

    def back(dyf, wt):
        z = torch.zeros(B, T, F, c, device=dev, requires_grad=True)
        return torch.autograd.grad(_conv_ref(z, wt, stride, pad, To), z, dyf)[0] * live

    for z in (None, torch.randn(B, T, F, c, device=dev).to(bf)):
        dx = torch.full((B, T, F, c), float("nan"), device=dev, dtype=bf)
        sums = torch.ones(c, device=dev)
        fe._conv(dy, w.permute(1, 2, 3, 0).reshape(c, 9 * n).contiguous(), None, z, dx, lens_in, lens_out, cu, None, None, B, T, To, F, n, c, stride, pad,
                 n_frames, True, sums)
        ref, mag = back(full, wf), back(full.abs(), wf.abs())
        if z is not None:
            ref, mag = ref * (z > 0), mag * (z > 0)
        assert ((dx.float() - ref).abs() <= 2.0**-8 * ref.abs() + 9 * n * 2.0**-24 * mag).all()
        cols = dx.double().view(-1, c)
        assert ((sums.double() - 1 - cols.sum(0)).abs() <= (cols.shape[0] + 1) * 2.0**-24 * (1 + cols.abs().sum(0))).all()

    dyp = torch.zeros(B, To, F, n, device=dev)
    dyp[pick] = dy.float().view(-1, F, n)
    dw = fe._conv_wgrad(x, dy, lens_in, row_batch, row_pos, B, T, To, F, c, n, stride, pad, n_frames)

    def filt(xf, dyf):  # in 64 bits, as the bound is that of one fp32 sum over all positions
        wt = torch.zeros(n, c, 3, 3, device=dev, dtype=torch.float64, requires_grad=True)
        return torch.autograd.grad(_conv_ref(xf.double(), wt, stride, pad, To), wt, dyf.double())[0].permute(0, 2, 3, 1).reshape(n, 9 * c)

    ref, mag = filt(xm, dyp), filt(xm.abs(), dyp.abs())
    assert ((dw.double() - ref).abs() <= n_frames * F * 2.0**-24 * mag).all()


def test_conv3x3_general_path_stays():
    """other channel counts and feature counts that are no multiple of 8 keep their patch matrices"""
    from returnn_b200.ops import _lib

    if _lib.get_lib() is None:
        pytest.skip("library not built")
    from returnn_b200.ops import frontend_native as fe

    assert not fe._implicit(40, 8, 16) and not fe._implicit(36, 32, 64) and not fe._implicit(88, 32, 64) and not fe._implicit(40, 32, 128)
