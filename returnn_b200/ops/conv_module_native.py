"""
Binding of the fused conv-module kernels (``csrc/conv_module.cu``): GLU + depthwise conv + BatchNorm (statistics over
the valid frames) + SiLU on packed rows, forward and backward. The per-CTA partial sums of the reductions (BatchNorm
statistics, dgamma/dbeta, dfilter) live in scratch buffers allocated per call.
"""

from __future__ import annotations
import ctypes
import torch
from . import _lib, nodes

_vp, _i32, _i64, _f32 = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float
_TT = 32


def available(x) -> bool:
    """library present with the entry points"""
    lib = _lib.get_lib()
    return lib is not None and hasattr(lib, "rb200_glu_dwconv_fwd") and x.is_cuda and x.dtype == torch.bfloat16


def supports(channels: int, kernel: int) -> bool:
    """shapes handled: channels multiple of 64 (and 256 % (C/8) == 0 for the BN backward), up to 64 taps"""
    groups = channels // 8
    return channels % 64 == 0 and 1 <= kernel <= 64 and groups <= 256 and 256 % groups == 0


def _p(t):
    return None if t is None else t.data_ptr()


class _ConvModuleFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, filt, bias, gamma, beta, running_mean, running_var, row_batch, row_pos, lens, eps, momentum, training):
        N, C2 = x.shape
        C = C2 // 2
        K = filt.shape[-1]
        dev = x.device
        x = x.contiguous()
        f32 = filt.reshape(C, K).float().contiguous()
        b32 = bias.float().contiguous() if bias is not None else None
        g32 = gamma.float().contiguous() if gamma is not None else None
        be32 = beta.float().contiguous() if beta is not None else None
        n_tiles = (N + _TT - 1) // _TT
        y = torch.empty(N, C, dtype=torch.bfloat16, device=dev)
        own_stats = training or running_mean is None
        part = torch.empty(n_tiles * 2 * C, dtype=torch.float32, device=dev) if own_stats or K > 32 else None
        stats = torch.empty(2, C, dtype=torch.float32, device=dev)  # mean, 1 / deviation
        if not own_stats:
            stats[0].copy_(running_mean.float())
            stats[1].copy_(torch.rsqrt(running_var.float() + eps))
        upd = training and running_mean is not None
        z = torch.empty(N, C, dtype=torch.bfloat16, device=dev)
        fn = _lib.bind("rb200_conv_module_fwd", [_vp] * 14 + [_i32] * 5 + [_f32, _f32, _vp])
        _lib.check(fn(x.data_ptr(), f32.data_ptr(), _p(b32), _p(g32), _p(be32), row_batch.data_ptr(), row_pos.data_ptr(), lens.data_ptr(), y.data_ptr(),
                      z.data_ptr(), _p(part), stats.data_ptr(), running_mean.data_ptr() if upd else None, running_var.data_ptr() if upd else None,
                      N, lens.shape[0], C, K, 1 if own_stats else 0, eps, momentum, _lib.stream_ptr()), "conv_module_fwd")
        _lib.count_launch(2 + (own_stats and (2 if K <= 32 else 1)))
        ctx.save_for_backward(x, f32, y, stats, g32, be32, row_batch, row_pos, lens)
        ctx.meta = (N, C, K, training, bias is not None, gamma is not None, beta is not None, filt.shape, filt.dtype,
                    bias.dtype if bias is not None else None, gamma.dtype if gamma is not None else None, beta.dtype if beta is not None else None)
        return z

    @staticmethod
    def backward(ctx, dz):
        x, f32, y, stats, g32, be32, row_batch, row_pos, lens = ctx.saved_tensors
        N, C, K, training, has_bias, has_gamma, has_beta, fshape, fdtype, bdtype, gdtype, bedtype = ctx.meta
        dev = dz.device
        dz = dz.contiguous()
        s = _lib.stream_ptr()
        n_tiles_a = min(296, max(1, (N + 15) // 16))
        ds = torch.empty(N, C, dtype=torch.bfloat16, device=dev)
        # the sums of the two passes, one after the other in the same scratch
        part = torch.empty(max(n_tiles_a * 2 * C, (N + _TT - 1) // _TT * C * (K + 1)), dtype=torch.float32, device=dev)
        sum_ds = torch.empty(C, dtype=torch.float32, device=dev)
        sum_ds_yh = torch.empty(C, dtype=torch.float32, device=dev)
        dx = torch.empty_like(x)
        dfilt = torch.empty(C, K, dtype=torch.float32, device=dev)
        dbias = torch.empty(C, dtype=torch.float32, device=dev) if has_bias else None
        if training:
            fn = _lib.bind("rb200_conv_module_bwd", [_vp] * 12 + [_i32] + [_vp] * 5 + [_i32] * 4 + [_vp])
            _lib.check(fn(x.data_ptr(), y.data_ptr(), dz.data_ptr(), stats.data_ptr(), f32.data_ptr(), _p(g32), _p(be32), row_batch.data_ptr(),
                          row_pos.data_ptr(), lens.data_ptr(), ds.data_ptr(), part.data_ptr(), n_tiles_a, sum_ds.data_ptr(), sum_ds_yh.data_ptr(),
                          dx.data_ptr(), dfilt.data_ptr(), _p(dbias), N, lens.shape[0], C, K, s), "conv_module_bwd")
            _lib.count_launch(5)
        else:
            mean, rstd = stats
            fn = _lib.bind("rb200_bn_silu_bwd", [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i32, _vp, _vp, _i64, _i32, _i32, _vp])
            _lib.check(fn(y.data_ptr(), dz.data_ptr(), mean.data_ptr(), rstd.data_ptr(), _p(g32), _p(be32), ds.data_ptr(), part.data_ptr(),
                          n_tiles_a, sum_ds.data_ptr(), sum_ds_yh.data_ptr(), N, C, 0, s), "bn_silu_bwd")
            # eval statistics are constants: dy = gamma * rstd * ds
            scale = rstd * (g32 if g32 is not None else 1.0)
            ds = (ds.float() * scale).to(torch.bfloat16)
            fn = _lib.bind("rb200_glu_dwconv_bwd", [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i32, _i32, _i32, _i32, _vp])
            _lib.check(fn(x.data_ptr(), ds.data_ptr(), f32.data_ptr(), row_batch.data_ptr(), row_pos.data_ptr(), lens.data_ptr(), dx.data_ptr(),
                          part.data_ptr(), dfilt.data_ptr(), _p(dbias), N, lens.shape[0], C, K, s), "glu_dwconv_bwd")
            _lib.count_launch(4)
        return (dx, dfilt.reshape(fshape).to(fdtype), dbias.to(bdtype) if has_bias else None,
                sum_ds_yh.to(gdtype) if has_gamma else None, sum_ds.to(bedtype) if has_beta else None,
                None, None, None, None, None, None, None, None)


def glu_dwconv_bn_silu(x, filt, bias, bn, pack, *, training):
    """fused path; ``bn`` is the rf.BatchNorm module (its running statistics are updated in place in training)"""
    gamma = bn.gamma.raw_tensor if bn.affine else None
    beta = bn.beta.raw_tensor if bn.affine else None
    rm = bn.running_mean.raw_tensor if bn.running_mean is not None else None
    rv = bn.running_variance.raw_tensor if bn.running_variance is not None else None
    mod = nodes.active() if training else None
    if mod is not None:
        return mod.conv_module(x, filt, bias, gamma, beta, rm, rv, pack.row_batch, pack.row_pos, pack.lens, bn.eps, bn.momentum)
    return _ConvModuleFn.apply(x, filt, bias, gamma, beta, rm, rv, pack.row_batch, pack.row_pos, pack.lens, float(bn.eps), float(bn.momentum), bool(training))
