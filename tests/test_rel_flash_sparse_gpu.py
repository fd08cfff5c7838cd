"""Backward pass of rel-pos attention that leaves out padding: buffers full of NaN give the position gradient and the valid rows of the whole form, with
probabilities recomputed (what the layer calls) and saved (what the encoder executor calls), without and with dropout."""

import ctypes

import pytest
import torch

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("lens,H", [([1], 1), ([64, 65, 0, 128], 2), ([320, 7, 201], 3), ([129, 1, 1, 1, 1, 1, 1, 190], 8), ([512, 300, 449], 2)])
@pytest.mark.parametrize("saved,p", [(False, 0.0), (False, 0.25), (True, 0.0), (True, 0.25)])
def test_sparse_padding(lens, H, saved, p):
    from returnn_b200.ops import _lib, gemm as G

    dev, bf, HD, B, L = "cuda", torch.bfloat16, H * 64, len(lens), max(lens)
    Lp, R = (L + 63) // 64 * 64, 2 * L - 1
    torch.manual_seed(L + H)
    n = torch.tensor(lens, dtype=torch.int32, device=dev)
    valid = torch.arange(Lp, device=dev)[None] < n[:, None]
    qu, qv, k, v, do = ((torch.randn(B, Lp, HD, device=dev) * valid[..., None]).to(bf) for _ in range(5))
    pos, o = torch.randn(R, HD, device=dev).to(bf), torch.randn(B, Lp, HD, device=dev)
    lse = torch.full((B, H, Lp), 12.0, device=dev)
    keep = torch.randint(-2**31, 2**31, (B, H, Lp, 4 * ((Lp + 127) // 128)), dtype=torch.int32, device=dev)
    w = torch.softmax(torch.randn(B, H, Lp, Lp, device=dev).masked_fill(~valid[:, None, None, :], -1e9), -1).to(bf)
    wd = (w * (torch.rand(B, H, Lp, Lp, device=dev) >= p) / (1 - p)).to(bf)
    vp, i32, f32, i64 = ctypes.c_void_p, ctypes.c_int, ctypes.c_float, ctypes.c_longlong
    geo = (ctypes.c_int * 2)()
    _lib.check(_lib.bind("rb200_rel_flash_band", [i32, i32, vp, vp])(Lp, L - 1, ctypes.addressof(geo), ctypes.addressof(geo) + 4), "band")
    width, st, s = geo[1], G.status_tensor(n.device).data_ptr(), _lib.stream_ptr()
    slices = _lib.bind("rb200_rel_flash_slices", [i64, i32, i32])(B * Lp, width, H)
    dpos = _lib.bind("rb200_rel_flash_dpos", [vp, vp, vp, vp, i32, i32, i32, i32, f32, i32, vp, vp])
    res = []
    for name in ("rb200_rel_flash_bwd", "rb200_rel_flash_bwd_sparse"):
        dqu, dqv, band = (torch.full(z, float("nan"), device=dev, dtype=bf) for z in ((B, Lp, HD), (B, Lp, HD), (H, B, Lp, width)))
        pw, ds = wd.clone() if saved else torch.zeros_like(w), torch.zeros_like(w)
        fn = _lib.bind(name, [vp] * 16 + [i32] * 5 + [f32, f32, vp, vp])
        _lib.check(fn(qu.data_ptr(), qv.data_ptr(), k.data_ptr(), v.data_ptr(), pos.data_ptr(), o.data_ptr(), do.data_ptr(), dqu.data_ptr(), dqv.data_ptr(),
                      w.data_ptr() if saved else None, pw.data_ptr(), ds.data_ptr(), band.data_ptr(), None if saved else lse.data_ptr(),
                      None if saved else keep.data_ptr(), n.data_ptr(), B, H, Lp, R, L - 1, 0.125, p, st, s), name)
        parts = []
        for m in sorted({1, slices, B}):
            part = torch.full((m, width, HD), float("nan"), device=dev, dtype=torch.float32 if m > 1 else bf)
            _lib.check(dpos(band.data_ptr(), qv.data_ptr(), part.data_ptr(), n.data_ptr(), B, H, Lp, L - 1, 0.125, m, st, s), "dpos")
            parts.append(part)
        G.check_status()
        res.append((dqu[valid], dqv[valid], pw, ds, *parts))
    for a, b in zip(*res):
        assert torch.isfinite(b).all() and torch.equal(a, b)
