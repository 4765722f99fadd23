"""Autograd nodes in C++ (``csrc/host_ops.cpp``) against the autograd functions in Python that call the same kernels: the same bits, the same
refusals, and nothing taken that only the Python form shows to hooks, transforms and modes.  Where gradients are summed with atomics (dQ of
attention, the norm's weight above 8192 columns) the order of the additions differs from run to run, in either form."""
import threading

import pytest
import torch

from lightron_b200.ops import functional as OF, native

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16


@pytest.fixture(autouse=True)
def _loaded():
    assert native.host_ops() is not None, "the extension module of the autograd nodes is missing"


def _t(*shape, seed=0, scale=1.0, grad=True):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(BF).requires_grad_(grad)


def _same(a, b, tol=None):
    assert (a is None) == (b is None)
    if a is None:
        return
    assert a.shape == b.shape and a.dtype == b.dtype and a.stride() == b.stride()
    if tol is None:
        assert torch.equal(a, b)
    else:
        assert (a.float() - b.float()).norm() <= tol * b.float().norm() + 1e-12


def _both(monkeypatch, fn, taken=True):
    """``fn()`` with the nodes and without; ``taken``: whether the nodes have to be the ones that ran."""
    host = native.host_ops()
    n0 = host.launches()
    new = fn()
    torch.cuda.synchronize()
    assert (host.launches() > n0) == taken
    with monkeypatch.context() as m:
        m.setattr(native, "_HOST", None)
        n0 = host.launches()
        old = fn()
        torch.cuda.synchronize()
        assert host.launches() == n0
    return new, old


def _grads(out, inputs, dy):
    outs = out if isinstance(out, tuple) else (out,)
    need = [t for t in inputs if t.requires_grad]
    if not need:
        return []
    return torch.autograd.grad(outs, need, dy, allow_unused=True)


@pytest.mark.parametrize("shape,widths", [((1, 8), (8,)), ((2, 24, 64), (16, 8, 8)), ((300, 256), (512,)), ((70, 264), (512, 136, 136)), ((8, 200, 512), (512, 256, 256))])
@pytest.mark.parametrize("need", [(True, True), (True, False), (False, True), (False, False)])
@pytest.mark.parametrize("form", ["dense", "expanded", "transposed"])
def test_linear(monkeypatch, shape, widths, need, form):
    def fn():
        x = _t(*shape, seed=1, grad=need[0])
        buf = _t(sum(widths), shape[-1], seed=2, scale=0.1, grad=False)
        ws, off = [], 0
        for n in widths:
            ws.append(buf[off:off + n].detach().requires_grad_(need[1]))
            off += n
        y = OF.linear(x, *ws)
        dy = {"dense": lambda: _t(*y.shape, seed=3, grad=False), "expanded": lambda: _t(1, seed=3, grad=False).expand(y.shape),
              "transposed": lambda: _t(*y.shape[:-2], y.shape[-1], y.shape[-2], seed=3, grad=False).transpose(-1, -2)}[form]()
        return [y.detach(), *_grads(y, [x, *ws], dy)]
    for a, b in zip(*_both(monkeypatch, fn)):
        _same(a, b)


@pytest.mark.parametrize("T,K,I", [(1, 8, 8), (8, 8, 8), (37, 264, 136), (104, 264, 136), (512, 512, 1408), (1531, 512, 1408)])
@pytest.mark.parametrize("need", [(1, 1, 1, 1), (1, 0, 0, 0), (0, 0, 0, 1), (0, 1, 1, 0), (0, 0, 0, 0)])
def test_swiglu_mlp(monkeypatch, T, K, I, need):
    def fn():
        x, buf = _t(T, K, seed=1, grad=False), _t(2 * I, K, seed=2, scale=0.1, grad=False)
        ts = [x, buf[:I], buf[I:], _t(K, I, seed=3, scale=0.1, grad=False)]
        ts = [t.detach().requires_grad_(bool(n)) for t, n in zip(ts, need)]
        y = OF.swiglu_mlp(*ts)
        return [y.detach(), *_grads(y, ts, _t(T, K, seed=4, grad=False))]
    for a, b in zip(*_both(monkeypatch, fn)):
        _same(a, b)


@pytest.mark.parametrize("shape", [(1, 8), (3, 33, 264), (300, 2048), (9, 8200)])
@pytest.mark.parametrize("res,used", [(False, "y"), (True, "hy"), (True, "h"), (True, "y")])
def test_rmsnorm(monkeypatch, shape, res, used):
    def fn():
        x, r, w = _t(*shape, seed=1), _t(*shape, seed=2), _t(shape[-1], seed=3)
        if not res:
            y = OF.rmsnorm(x, w, 1e-5)
            return [y.detach(), *_grads(y, [x, w], _t(*shape, seed=4, grad=False))]
        h, y = OF.add_rmsnorm(x, r, w, 1e-5)
        outs = tuple({"h": h, "y": y}[c] for c in used)
        return [h.detach(), y.detach(), *_grads(outs, [x, r, w], tuple(_t(*shape, seed=4 + i, grad=False) for i in range(len(outs))))]
    new, old = _both(monkeypatch, fn)
    for i, (a, b) in enumerate(zip(new, old)):
        # above 8192 columns the weight gradient is summed with atomics in fp32 and rounded to bf16 once: 2^-8 and some
        _same(a, b, tol=5e-3 if shape[-1] > 8192 and i == len(new) - 1 else None)


@pytest.mark.parametrize("bwd", ["tc", "mma"])
@pytest.mark.parametrize("form", ["dense", "fused", "heads_first"])
@pytest.mark.parametrize("B,Sq,Sk,hq,hkv,d,causal", [(1, 1, 1, 1, 1, 64, True), (2, 129, 200, 4, 2, 128, True), (3, 65, 31, 2, 1, 64, False)])
def test_attention(monkeypatch, B, Sq, Sk, hq, hkv, d, causal, form, bwd):
    monkeypatch.setenv("LIGHTRON_FA_BWD", bwd)
    def make(S, h, seed):
        if form == "fused":
            return _t(B, S, h + 2, d, seed=seed, grad=False)[:, :, 1:1 + h].detach().requires_grad_()
        if form == "heads_first":
            return _t(B, h, S, d, seed=seed, grad=False).transpose(1, 2).detach().requires_grad_()
        return _t(B, S, h, d, seed=seed)
    def fn():
        q, k, v = make(Sq, hq, 1), make(Sk, hkv, 2), make(Sk, hkv, 3)
        o = OF.flash_attention(q, k, v, causal)
        return [o.detach(), *_grads(o, [q, k, v], _t(B, Sq, hq, d, seed=4, grad=False))]
    for i, (a, b) in enumerate(zip(*_both(monkeypatch, fn))):
        _same(a, b, tol=None if i == 0 else 2e-3)       # gradients: fp32 atomics, then one rounding to bf16 (2^-9 at most on few elements)


@pytest.mark.parametrize("B,S,hq,hkv,d", [(1, 1, 1, 1, 64), (2, 130, 4, 2, 64), (2, 65, 2, 1, 128)])
@pytest.mark.parametrize("pos", [None, torch.int32, torch.int64])
def test_rope_attention(monkeypatch, B, S, hq, hkv, d, pos):
    cos, sin = _tables(2 * S, d)
    p = None if pos is None else torch.arange(S, device=DEV, dtype=pos).flip(0) + S // 2
    def fn():
        qkv = _t(B * S, (hq + 2 * hkv) * d, seed=1)
        o = OF.rope_attention_qkv(qkv * 1, cos, sin, p, B, S, hq, hkv, d)
        return [o.detach(), *_grads(o, [qkv], _t(B * S, hq * d, seed=2, grad=False))]
    for i, (a, b) in enumerate(zip(*_both(monkeypatch, fn))):
        _same(a, b, tol=None if i == 0 else 2e-3)


def _tables(n, d):
    f = torch.arange(n, device=DEV).float()[:, None] / 10000.0 ** (torch.arange(0, d, 2, device=DEV).float() / d)
    return f.cos().contiguous(), f.sin().contiguous()


@pytest.mark.parametrize("shape,V,H,v0", [((1,), 1, 8, 0), ((3, 41), 123, 264, 0), ((2, 64), 200, 2048, 50)])
def test_embedding(monkeypatch, shape, V, H, v0):
    n = torch.Size(shape).numel()
    tok = torch.randperm(max(n, V), device=DEV)[:n].view(shape)         # every id once: no two additions meet
    def fn():
        w = _t(V, H, seed=1)
        y = OF.embedding(tok, w, v0)
        return [y.detach(), *_grads(y, [w], _t(*shape, H, seed=2, grad=False))]
    for a, b in zip(*_both(monkeypatch, fn)):
        _same(a, b)


@pytest.mark.parametrize("T,V,ignore", [(1, 8, -100), (37, 1000, -100), (64, 32000, 7)])
def test_cross_entropy(monkeypatch, T, V, ignore):
    tgt = torch.randint(0, V, (T,), device=DEV)
    tgt[::3] = ignore
    def fn():
        x = _t(T, V, seed=1)
        loss = OF.cross_entropy(x * 1, tgt, n_valid_total=max(T - (T + 2) // 3, 1), ignore_index=ignore)
        return [loss.detach(), *_grads(loss, [x], torch.tensor(0.5, device=DEV))]
    for i, (a, b) in enumerate(zip(*_both(monkeypatch, fn))):
        _same(a, b, tol=1e-6 if i == 0 else None)       # the loss is a sum over blocks in the order of their arrival


def test_what_is_not_plain_goes_the_old_way(monkeypatch):
    w = _t(16, 64, seed=2)
    tgt = torch.randint(0, 32, (8,), device=DEV)
    for fn in (lambda: OF.linear(_t(24, 128)[:, :64], w), lambda: OF.linear(_t(24, 64), w, _t(16, 64, seed=3)), lambda: OF.linear(_t(8, 64), _t(4, 64)),
               lambda: OF.linear(_t(8, 64).float(), w.float()), lambda: OF.rmsnorm(_t(64, 24).t(), _t(64), 1e-5),
               lambda: OF.flash_attention(*(_t(1, 8, 2, 32, seed=i) for i in range(3))),
               lambda: OF.cross_entropy(_t(8, 32, grad=False), tgt), lambda: OF.embedding(tgt.int().long()[::2], _t(32, 64))):
        new, old = _both(monkeypatch, fn, taken=False)
        assert torch.allclose(new.float(), old.float(), rtol=1e-5)
    for fn, err in ((lambda: OF.cross_entropy(_t(8, 32), tgt[:4], n_valid_total=4), ValueError), (lambda: OF.linear(_t(8, 64), _t(16, 56)), AssertionError)):
        with pytest.raises(err):
            fn()
    w.grad, w._lb_direct_grad = torch.zeros_like(w), True               # a weight of the optimizer's arena: accumulated by the GEMM
    _both(monkeypatch, lambda: OF.linear(_t(8, 64), w).sum().backward(), taken=False)
    assert w.grad.abs().sum() > 0


def test_a_mark_without_truth_value_goes_the_old_way(monkeypatch):
    """The attribute that marks a weight of the arena may be anything: the node declines, without an error of its own."""
    class Unclear:
        def __bool__(self):
            raise ValueError("neither")
    w = _t(16, 64, seed=2)
    w._lb_direct_grad = Unclear()
    new, old = _both(monkeypatch, lambda: OF.linear(_t(8, 64), w).detach(), taken=False)
    assert torch.equal(new, old)


def test_errors_are_the_same():
    with pytest.raises(native.NativeError, match="lb_rmsnorm_fwd failed: unsupported shape"):
        OF.rmsnorm(_t(4, 12), _t(12), 1e-5)
    x, w = _t(8, 64), _t(16, 64, seed=1)
    y = OF.linear(x, w)
    with torch.no_grad():
        w.mul_(2)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.sum().backward()
    y = OF.linear(x, w)
    y.sum().backward()
    with pytest.raises(RuntimeError, match="second time"):
        y.sum().backward()


def test_observers_see_what_they_did(monkeypatch):
    x, w = _t(8, 64), _t(16, 64, seed=1)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t.cpu(), lambda t: t.to(DEV)):
        y = OF.linear(x, w)
    assert packed == [x.shape, w.shape]
    y.sum().backward()
    assert torch.equal(x.grad, torch.autograd.grad(OF.linear(x, w).sum(), x)[0])

    from torch.utils._python_dispatch import TorchDispatchMode

    class Count(TorchDispatchMode):
        n = 0
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            Count.n += 1
            return func(*args, **(kwargs or {}))
    host = native.host_ops()
    n0 = host.launches()
    with Count():
        OF.linear(x, w)
    assert Count.n > 0 and host.launches() == n0
    with torch.inference_mode():
        a = OF.linear(x, w)
    with torch.no_grad():
        b = OF.linear(x, w)
    assert host.launches() == n0 + 2 and a.is_inference() and not b.requires_grad and torch.equal(a, b)
    n0 = host.launches()
    with torch.autograd.forward_ad.dual_level():
        with pytest.raises((RuntimeError, NotImplementedError)):
            OF.linear(torch.autograd.forward_ad.make_dual(x.detach(), torch.ones_like(x)), w)
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: OF.linear(t, w).float().sum())(x.detach())
    assert host.launches() == n0


def _strided(t):
    """The same values two elements apart."""
    buf = torch.zeros(*t.shape, 2, dtype=t.dtype, device=t.device)
    buf[..., 0] = t
    return buf[..., 0]


def _op_cases():
    """name -> (op, its differentiable inputs, its output's shape)"""
    cos, sin = _tables(48, 64)
    pos = torch.arange(48, device=DEV, dtype=torch.int32).flip(0)
    tok, tgt = torch.arange(24, device=DEV) % 16, torch.arange(24, device=DEV)
    qkv = lambda: [_t(2, 24, h, 64, seed=i) for i, h in enumerate((4, 2, 2))]
    return {
        "linear": (OF.linear, lambda: [_t(24, 64, seed=1), _t(16, 64, seed=2)], (24, 16)),
        "rmsnorm": (lambda x, w: OF.rmsnorm(x, w, 1e-5), lambda: [_t(24, 64, seed=1), _t(64, seed=2)], (24, 64)),
        "add_rmsnorm": (lambda x, r, w: OF.add_rmsnorm(x, r, w, 1e-5)[1], lambda: [_t(24, 64, seed=1), _t(24, 64, seed=2), _t(64, seed=3)], (24, 64)),
        "attention": (OF.flash_attention, qkv, (2, 24, 4, 64)),
        "rope_attention": (lambda t: OF.rope_attention_qkv(t * 1, cos, sin, pos, 1, 48, 4, 2, 64), lambda: [_t(48, 512, seed=1)], (48, 256)),
        "embedding": (lambda w: OF.embedding(tok, w), lambda: [_t(32, 64, seed=1)], (24, 64)),
        "cross_entropy": (lambda x: OF.cross_entropy(x * 1, tgt, n_valid_total=24), lambda: [_t(24, 64, seed=1)], ()),
    }


@pytest.mark.parametrize("name", ["linear", "rmsnorm", "add_rmsnorm", "attention", "rope_attention", "embedding", "cross_entropy"])
def test_saved_tensors_come_back_otherwise(name):
    """A copy, and a copy with other strides: the same gradients (attention: dQ is summed with atomics).  Other sizes or types, and batched
    gradients, which have no memory: refused."""
    op, make, out = _op_cases()[name]
    host = native.host_ops()
    dy = _t(*out, seed=9, grad=False) if out else torch.ones((), device=DEV)
    n0 = host.launches()

    def grads(unpack):
        ins = make()
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            y = op(*ins)
        return torch.autograd.grad(y, ins, dy)
    want = grads(lambda t: t)
    for unpack in (lambda t: t.clone(), lambda t: _strided(t)):
        for g, w in zip(grads(unpack), want):
            _same(g, w, tol=2e-3 if "attention" in name else None)
    ins = make()
    with torch.autograd.graph.save_on_cpu():
        y = op(*ins)
    for g, w in zip(torch.autograd.grad(y, ins, dy), want):
        _same(g, w, tol=2e-3 if "attention" in name else None)
    for unpack in (lambda t: t[:-1], lambda t: t.double(), lambda t: t.cpu()):
        with pytest.raises(RuntimeError, match="saved for backward"):
            grads(unpack)
    ins = make()
    with pytest.raises(RuntimeError):
        torch.autograd.grad(op(*ins), ins, dy.expand(3, *dy.shape), is_grads_batched=True)
    torch.cuda.synchronize()
    assert host.launches() > n0


@pytest.mark.parametrize("op,n", [(OF.linear, 2), (OF.linear, 3), (OF.swiglu_mlp, 3)])
def test_adjacent_weights_come_back_apart(monkeypatch, op, n):
    """The data gradient reads the adjacent weights as one matrix: refused where the hooks give each its own memory, in either form.  What
    does not need it, and weights that are still adjacent (recomputation), give the same gradients."""
    from torch.utils.checkpoint import checkpoint

    def make(need_x=True):
        buf = _t(n * 40, 64, seed=2, scale=0.1, grad=False)
        ws = [buf[i * 40:i * 40 + 40].detach().requires_grad_() for i in range(n if op is OF.linear else 2)]
        if op is OF.swiglu_mlp:
            ws.append(_t(64, 40, seed=3, scale=0.1))
        return [_t(37, 64, seed=1).requires_grad_(need_x), *ws]
    dy = _t(*op(*make()).shape, seed=4, grad=False)

    def grads(need_x, ctx, call=op):
        ins = make(need_x)
        with ctx:
            y = call(*ins)
        return torch.autograd.grad(y, ins if need_x else ins[1:], dy)
    import contextlib
    want = grads(True, contextlib.nullcontext())
    assert native.host_ops() is not None
    for g, w in zip(grads(True, contextlib.nullcontext(), lambda *a: checkpoint(op, *a, use_reentrant=False)), want):
        _same(g, w)
    apart = (torch.autograd.graph.save_on_cpu, lambda: torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t.clone()))
    for ctx in apart:
        with pytest.raises(RuntimeError, match="separate tensors"):
            grads(True, ctx())
        for g, w in zip(grads(False, ctx()), want[1:]):
            _same(g, w)
    with monkeypatch.context() as m:
        m.setattr(native, "_HOST", None)
        for ctx in apart:
            with pytest.raises(RuntimeError, match="out of bounds for storage"):
                grads(True, ctx())
    torch.cuda.synchronize()


def test_threads_and_streams():
    x, w = _t(64, 512), _t(512, 512, seed=1, scale=0.05)
    want = OF.linear(x.detach(), w.detach())
    torch.cuda.synchronize()
    bad = []

    def work(i):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(20):
                a = x.detach().requires_grad_()
                y = OF.linear(a, w.detach())
                y.sum().backward()
                if not torch.equal(y, want) or not torch.isfinite(a.grad).all():
                    bad.append(i)
            s.synchronize()
    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad
