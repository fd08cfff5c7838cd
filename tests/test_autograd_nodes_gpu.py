"""The autograd nodes in C++ against the Python functions of the same operators: results and gradients equal, over the forms that the calls accept."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _both(monkeypatch, call, inputs, grad_of):
    """results and gradients of `call(*inputs)` with the nodes and without them"""
    from returnn_b200.ops import nodes

    assert nodes.active() is not None, "the extension is not built"
    res = []
    for python in (False, True):
        with monkeypatch.context() as m:
            if python:
                m.setattr(nodes, "active", lambda: None)
            leaves = [x.detach().clone().requires_grad_(x.requires_grad) if x is not None else None for x in inputs]
            y = call(*leaves)
            wanted = [x for x in leaves if x is not None and x.requires_grad]
            g = torch.autograd.grad(y, wanted, grad_of(y)) if wanted else []
            res.append((y, *g))
    return res


def _same(a, b):
    for x, y in zip(a, b):
        assert x.shape == y.shape and x.dtype == y.dtype and x.device == y.device
        assert torch.equal(x, y), float((x.float() - y.float()).abs().max())


def _rand(*shape, dtype=torch.bfloat16, grad=True, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + sum(shape))
    return torch.randn(*shape, generator=g, device="cuda").to(dtype).requires_grad_(grad)


@pytest.mark.parametrize("shape,dtype,w_dtype,beta,rms", [
    ((7, 3, 64), torch.bfloat16, torch.bfloat16, True, False), ((33, 512), torch.bfloat16, torch.float32, False, True),
    ((5, 1024), torch.float32, torch.float32, True, False), ((1, 8), torch.float32, torch.bfloat16, True, True)])
def test_layer_norm(monkeypatch, shape, dtype, w_dtype, beta, rms):
    from returnn_b200.ops import layer_norm as L

    fn = L.rms_norm if rms else L.layer_norm
    x = _rand(*shape, dtype=dtype)
    inputs = [x, _rand(shape[-1], dtype=w_dtype, seed=1), _rand(shape[-1], dtype=w_dtype, seed=2) if beta else None]
    a, b = _both(monkeypatch, lambda x, g, b: fn(x.transpose(0, 1).transpose(0, 1), g, b, 1e-5), inputs, lambda y: torch.ones_like(y) * 0.5)
    _same(a[:2], b[:2])
    for p, q in zip(a[2:], b[2:]):  # parameter gradients are sums by atomics
        torch.testing.assert_close(p.float(), q.float(), rtol=2 ** -7 if w_dtype == torch.bfloat16 else 1e-5, atol=1e-4)


@pytest.mark.parametrize("shape,n,w_dtype,bias,act,grads", [
    ((3, 40, 64), 72, torch.float32, torch.float32, "silu", (1, 1, 1)), ((2048, 64), 64, torch.float32, torch.bfloat16, None, (0, 1, 1)),
    ((1, 512), 512, torch.bfloat16, None, "gelu", (1, 0, 0)), ((130, 64), 136, torch.bfloat16, torch.float16, "relu", (1, 1, 0)),
    ((64, 16), 8, torch.float32, torch.float32, "relu", (0, 0, 0)), ((70, 64), 72, torch.float32, torch.float32, "silu", (0, 0, 1)),
    ((70, 64), 72, torch.bfloat16, torch.bfloat16, "relu", (0, 0, 1))])
def test_linear(monkeypatch, shape, n, w_dtype, bias, act, grads):
    from returnn_b200.ops.gemm import linear_bf16

    inputs = [_rand(*shape, grad=bool(grads[0])), _rand(shape[-1], n, dtype=w_dtype, grad=bool(grads[1]), seed=1),
              _rand(n, dtype=bias, grad=bool(grads[2]), seed=2) if bias else None]
    a, b = _both(monkeypatch, lambda x, w, b: linear_bf16(x, w, b, act), inputs, lambda y: _rand(*y.shape, grad=False, seed=3))
    _same(a, b)


@pytest.mark.parametrize("start", [0, 1])
def test_relu_gradient_that_is_not_finite(monkeypatch, start):
    """zero where the activation is zero, also where the gradient there is not finite, and for gradients off the alignment of the kernel"""
    from returnn_b200.ops.gemm import linear_bf16

    x, w, b = _rand(40, 64), _rand(64, 72, dtype=torch.float32, seed=1), _rand(72, dtype=torch.float32, seed=2)
    off = linear_bf16(x, w, b, "relu").detach() == 0

    def grad(bad):
        dy = torch.zeros(start + off.numel(), dtype=torch.bfloat16, device="cuda")[start:].view_as(off)
        dy[off] = torch.tensor(bad, dtype=torch.bfloat16, device="cuda").repeat(off.numel())[: int(off.sum())]
        dy[~off] = 0.5
        return dy

    res = [_both(monkeypatch, lambda x, w, b: linear_bf16(x, w, b, "relu"), [x, w, b], lambda y: grad(bad))
           for bad in ([1.0], [float("inf"), float("nan"), float("-inf")])]
    for a, b in zip(*res):
        _same(a, b)


@pytest.mark.parametrize("lens,taps,affine,stats", [([5, 0, 33], 32, True, True), ([1], 7, False, True), ([40, 41], 33, True, False)])
def test_conv_module(monkeypatch, lens, taps, affine, stats):
    from types import SimpleNamespace as NS
    from returnn_b200.models.packing import PackInfo
    from returnn_b200.ops.conv_module import glu_dwconv_bn_silu

    C = 64
    pack = PackInfo(torch.tensor(lens, dtype=torch.int32), "cuda")
    running = []

    def call(x, f, b, g, be):
        mean, var = torch.zeros(C, device="cuda"), torch.ones(C, device="cuda")
        running.append((mean, var))
        bn = NS(affine=affine, eps=1e-3, momentum=0.1, gamma=NS(raw_tensor=g), beta=NS(raw_tensor=be),
                running_mean=NS(raw_tensor=mean) if stats else None, running_variance=NS(raw_tensor=var) if stats else None)
        return glu_dwconv_bn_silu(x, f, b, bn, pack, training=True)

    inputs = [_rand(pack.n, 2 * C), _rand(C, 1, taps, dtype=torch.float32), _rand(C, dtype=torch.float32, grad=False, seed=1)]
    inputs += [_rand(C, dtype=torch.float32, grad=affine, seed=s) for s in (2, 3)]
    a, b = _both(monkeypatch, call, inputs, lambda y: _rand(*y.shape, grad=False, seed=4))
    _same(a, b)
    _same(*running)


@pytest.mark.parametrize("B,Tq,Tk,H,causal,lens,drop,fused", [(2, 70, 70, 2, True, False, 0.0, True), (3, 5, 130, 1, False, True, 0.0, False),
                                                              (1, 1, 9, 4, False, False, 0.25, False), (2, 33, 33, 3, True, True, 0.1, True)])
def test_attention(monkeypatch, B, Tq, Tk, H, causal, lens, drop, fused):
    from returnn_b200.ops import elementwise
    from returnn_b200.ops.sdpa import sdpa_heads

    kl = torch.tensor([Tk - i * (Tk // 2) for i in range(B)], dtype=torch.int32, device="cuda").clamp(min=1) if lens else None
    seed = elementwise._seed_tensor(torch.device("cuda", 0))
    start = seed.clone()
    ends = []

    def call(*xs):
        seed.copy_(start)
        q, k, v = (xs[0][..., 64 * i: 64 * i + 64] for i in range(3)) if fused else xs
        y = sdpa_heads(q, k, v, k_lens=kl, causal=causal, dropout_p=drop)
        ends.append(seed.clone())
        return y

    inputs = [_rand(B, Tq, H, 192)] if fused else [_rand(B, Tq, H, 64), _rand(B, Tk, H, 64, dtype=torch.float32, seed=1).bfloat16().detach().requires_grad_(True),
                                                   _rand(B, Tk, H, 64, seed=2)]
    a, b = _both(monkeypatch, call, inputs, lambda y: _rand(*y.shape, grad=False, seed=3).transpose(1, 2).contiguous().transpose(1, 2))
    _same(a, b)
    assert torch.equal(*ends)


@pytest.mark.parametrize("dtype,smoothing,grad_only", [(torch.bfloat16, 0.1, False), (torch.float32, 0.0, False), (torch.float32, 0.2, True)])
def test_cross_entropy(monkeypatch, dtype, smoothing, grad_only):
    from returnn_b200.ops.softmax_ce import softmax_cross_entropy

    tgt = torch.arange(11, device="cuda") * 3
    a, b = _both(monkeypatch, lambda x: softmax_cross_entropy(x, tgt, smoothing, grad_only_smoothing=grad_only), [_rand(11, 100, dtype=dtype)],
                 lambda y: torch.linspace(-1, 1, 11, device="cuda"))
    _same(a, b)


def test_hooks_of_saved_tensors_and_released_graphs():
    from returnn_b200.ops.layer_norm import layer_norm

    x, g = _rand(9, 64), _rand(64, seed=1)
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(t.shape) or t.cpu(), lambda t: t.cuda()):
        y = layer_norm(x, g, None, 1e-5)
    assert len(seen) == 4
    (dx,) = torch.autograd.grad(y.sum(), [x])
    (ref,) = torch.autograd.grad(layer_norm(x, g, None, 1e-5).sum(), [x])
    assert torch.equal(dx, ref)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(y.sum(), [x])


def test_traced_programs_record_the_python_function():
    from returnn_b200.ops.layer_norm import layer_norm

    g = _rand(64, grad=False)
    traced = torch.jit.trace(lambda x: layer_norm(x, g, None, 1e-5), (_rand(9, 64, grad=False),), check_trace=False)
    x = _rand(9, 64, grad=False, seed=5)
    assert torch.equal(traced(x), layer_norm(x, g, None, 1e-5))


def _chain(x, w, b, g, v):
    """a layer norm, a linear layer, attention and a cross entropy"""
    from returnn_b200.ops.gemm import linear_bf16
    from returnn_b200.ops.layer_norm import layer_norm
    from returnn_b200.ops.sdpa import sdpa_heads
    from returnn_b200.ops.softmax_ce import softmax_cross_entropy

    B, T, _ = x.shape
    qkv = linear_bf16(layer_norm(x, g, None, 1e-5), w, b, "silu").view(B, T, 2, 192)
    y = sdpa_heads(qkv[..., :64], qkv[..., 64:128], qkv[..., 128:], causal=True).reshape(B * T, 128)
    return softmax_cross_entropy(linear_bf16(y, v, None, None), torch.arange(B * T, device="cuda") % 96, 0.1)


def _chain_inputs(seed):
    shapes = ((3, 50, 128), torch.bfloat16), ((128, 384), torch.float32), ((384,), torch.float32), ((128,), torch.float32), ((128, 96), torch.float32)
    return [_rand(*s, dtype=dt, seed=seed + i) for i, (s, dt) in enumerate(shapes)]


def _close(a, b):
    for x, y in zip(a, b):  # (the gradient of gamma is a sum by atomics)
        torch.testing.assert_close(x.float(), y.float(), rtol=1e-5, atol=1e-4)


def test_two_threads_and_streams_of_their_own():
    import threading

    want = []
    for t in range(2):
        x = _chain_inputs(10 * t)
        loss = _chain(*x)
        want.append((loss.detach(), *torch.autograd.grad(loss.sum(), x)))
    torch.cuda.synchronize()
    got, errors = [[], []], []

    def work(t):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(5):
                    x = _chain_inputs(10 * t)
                    loss = _chain(*x)
                    got[t].append((loss.detach(), *torch.autograd.grad(loss.sum(), x)))
                torch.cuda.current_stream().synchronize()
        except BaseException as exc:  # noqa: B902
            errors.append(exc)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for t in range(2):
        for res in got[t]:
            _close(res, want[t])


def test_second_backward_through_a_retained_graph():
    x = _chain_inputs(3)
    loss = _chain(*x)
    a = torch.autograd.grad(loss.sum(), x, retain_graph=True)
    b = torch.autograd.grad(loss.sum() * 2, x, retain_graph=True)
    c = torch.autograd.grad(loss.sum(), x)
    _close(a, c)
    for p, q in zip(a, b):  # a factor of two is exact in every rounding on the way
        torch.testing.assert_close(2 * p.float(), q.float(), rtol=1e-5, atol=2e-4)


@pytest.mark.parametrize("python", [False, True])
def test_function_transforms_are_refused(monkeypatch, python):
    """torch.func and forward mode: an error from the nodes as from the Python functions, not a result that leaves the operator out"""
    from returnn_b200.ops import nodes
    from returnn_b200.ops.layer_norm import layer_norm

    if python:
        monkeypatch.setattr(nodes, "active", lambda: None)
    x, g = _rand(4, 64, grad=False), _rand(64, grad=False, seed=1)
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: layer_norm(t, g, None, 1e-5).float().sum())(x)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda t: layer_norm(t, g, None, 1e-5))(x[:, None])
    with torch.autograd.forward_ad.dual_level(), pytest.raises((RuntimeError, NotImplementedError)):
        layer_norm(torch.autograd.forward_ad.make_dual(x, torch.ones_like(x)), g, None, 1e-5)
