"""With gradients off the ops call an autograd function's forward directly; everything that looks at autograd functions
still gets the function."""
import os
import subprocess
import sys

import pytest
import torch
import torch.autograd.forward_ad as fwAD

from lightron_b200.ops import functional as OF


class _Twice(torch.autograd.Function):
    applied = 0

    @staticmethod
    def forward(ctx, x, y):
        ctx.save_for_backward(x, y)
        ctx.shape = x.shape
        return 2 * x + y

    @staticmethod
    def backward(ctx, g):
        return 2 * g, g


@pytest.fixture
def wrapped(monkeypatch):
    calls = []
    real = _Twice.apply
    monkeypatch.setattr(_Twice, "apply", lambda *a: (calls.append(1), real(*a))[1])
    return calls


def test_gradients_on_uses_the_function(wrapped):
    x, y = torch.randn(3, requires_grad=True), torch.randn(3)
    out = OF._apply(_Twice, x, y)
    out.sum().backward()
    assert wrapped and torch.equal(x.grad, torch.full((3,), 2.0))
    saved = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: saved.append(t) or t, lambda t: t):
        OF._apply(_Twice, x, y)
    assert len(saved) == 2


@pytest.mark.parametrize("mode", [torch.no_grad, torch.inference_mode])
def test_gradients_off_gives_the_same_values(wrapped, mode):
    x, y = torch.randn(3, requires_grad=True), torch.randn(3)
    with mode():
        got = OF._apply(_Twice, x, y)
    assert not wrapped and not got.requires_grad and torch.equal(got, 2 * x.detach() + y)


def test_transforms_and_tangents_still_reach_the_function(wrapped):
    x, y = torch.randn(4, 3), torch.randn(4, 3)
    with torch.no_grad():
        with pytest.raises(RuntimeError):                       # no vmap rule: refused, not computed on wrappers
            torch.func.vmap(lambda a, b: OF._apply(_Twice, a, b))(x, y)
        assert wrapped
        wrapped.clear()
        with fwAD.dual_level():
            with pytest.raises(Exception):                      # no jvp rule: refused, the tangent is not dropped
                OF._apply(_Twice, fwAD.make_dual(x, torch.ones_like(x)), y)
        assert wrapped


def test_tracing_still_reaches_the_function(wrapped):
    x, y = torch.randn(3), torch.randn(3)
    with torch.no_grad():
        traced = torch.jit.trace(lambda a, b: OF._apply(_Twice, a, b), (x, y), check_trace=False)
    assert wrapped and torch.equal(traced(x, y), 2 * x + y)


def test_a_torch_without_the_private_names_uses_public_ones():
    """Neither the short path nor the stream handle is needed: without the names that they read, the public way is taken."""
    code = """
import torch
import torch.autograd.forward_ad
del torch.autograd.forward_ad._current_level
if hasattr(torch._C, "_cuda_getCurrentRawStream"): del torch._C._cuda_getCurrentRawStream
from lightron_b200.ops import functional as OF, native
class F(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        ctx.set_materialize_grads(False)        # only the real context has it
        return 2 * x
with torch.no_grad():
    assert torch.equal(OF._apply(F, torch.ones(2)), torch.full((2,), 2.0))
class S: cuda_stream = 7
torch.cuda.current_stream = S
assert native.stream_ptr() == 7
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("n", [3, 5, 1])
def test_targets_have_to_match_the_rows(monkeypatch, n):
    """The kernels read a target per row of logits: another number is refused before any of them is launched."""
    monkeypatch.setattr(OF.native, "use_native", lambda t: True)
    monkeypatch.setattr(OF.native, "stream_ptr", lambda: 0)
    calls = []
    monkeypatch.setattr(OF.native, "call", lambda *a: calls.append(a[0]))
    with pytest.raises(ValueError):
        OF.cross_entropy(torch.randn(4, 8), torch.zeros(n, dtype=torch.long))
    assert not calls
    OF.cross_entropy(torch.randn(4, 8), torch.zeros(2, 2, dtype=torch.long))
    assert calls == ["lb_ce_stats", "lb_ce_loss"]
