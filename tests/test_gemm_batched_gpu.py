"""Batched products with 64 columns on both sides of the rule that gives an SM two CTAs (more units than SMs), at the edges of the tiles."""

import pytest
import torch

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("lens,H", [([65, 1, 0, 64], 3), ([129, 128, 127, 1] * 12, 4), ([320, 7, 201], 40), ([513, 450], 70)])
@pytest.mark.parametrize("fp32", [False, True])
def test_transposed_product(lens, H, fp32):
    from returnn_b200.ops import attention_native as an

    torch.manual_seed(0)
    torch.backends.cuda.matmul.allow_tf32 = False
    B, Lp, dev = len(lens), (max(lens) + 63) // 64 * 64, "cuda"
    ln = torch.tensor(lens, dtype=torch.int32, device=dev)
    p = torch.randn(B * H * Lp, Lp, device=dev).bfloat16()
    do = torch.randn(B * Lp, H * 64, device=dev).bfloat16()
    out = torch.full((B * Lp, H * 64), 7.0, device=dev, dtype=torch.float32 if fp32 else torch.bfloat16)
    an._bgemm(p, do, out, m=Lp, n=64, k=Lp, a_mn=True, b_mn=True, lda=Lp, ldb=H * 64, ldc=H * 64, a_shape=(B * H * Lp, Lp), b_shape=(B * Lp, H * 64),
              offs=(H * Lp, Lp, 0, 0, Lp, 0, 0, 64, Lp * H * 64, 64), batch=B * H, heads=H, lens=ln, m_l=True, n_l=False, k_l=True, alpha=0.5, out_fp32=fp32)
    at = torch.arange(Lp, device=dev)
    rows = (at[None] < (ln[:, None] + 63) // 64 * 64).float()  # the contraction runs in blocks of 64 rows
    keys = (at[None] < ln[:, None])[:, :, None, None].expand(B, Lp, H, 64)
    a, b = p.view(B, H, Lp, Lp).float() * rows[:, None, :, None], do.view(B, Lp, H, 64).float()
    ref = 0.5 * torch.einsum("bhqk,bqhd->bkhd", a, b)
    mag = 0.5 * torch.einsum("bhqk,bqhd->bkhd", a.abs(), b.abs())
    got = out.view(B, Lp, H, 64).float()
    bound = Lp * 2.0**-23 * mag + (0.0 if fp32 else 2.0**-8) * ref.abs()  # order of the fp32 sums on both sides, one rounding
    assert ((got - ref).abs() <= bound)[keys].all()
    assert (got[~keys] == 7.0).all()  # rows past a sequence's length are not written
