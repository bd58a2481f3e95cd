"""The native autograd formula of hstu_jagged on Meta tensors: which inputs get gradients, what is saved, what tracing sees,
and what stays refused (the values are checked on the GPU, tests/test_gpu_backward.py)."""
import pytest
import torch

import ops_rec_b200

op = ops_rec_b200.ascendc.attention.hstu_jagged
OFF = torch.zeros(3, dtype=torch.int64, device="meta")


def qkv(grad=True):
    return [torch.empty(10, 2, 64, device="meta", dtype=torch.bfloat16).requires_grad_(grad) for _ in range(3)]


def plane(grad):
    return torch.empty(2, 2, 16, 16, device="meta", dtype=torch.bfloat16).requires_grad_(grad)


def call(delta, q, k, v, bias=None, mask=None):
    if delta:
        return op(q, k, v, mask, bias, 0, 16, 16, 0.0, OFF, OFF, None, None, 0, 0.1)
    return op(q, k, v, mask, bias, 0, 16, 0.0, OFF, None, None, 0, 0.1)


@pytest.mark.parametrize("delta", [False, True])
def test_gradients_reach_every_differentiable_input(delta):
    leaves = qkv() + [plane(True)]
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t, lambda t: t):
        out = call(delta, *leaves)
    grads = torch.autograd.grad(out, leaves, torch.empty_like(out))
    assert [g.shape for g in grads] == [t.shape for t in leaves]
    assert len(packed) == (6 if delta else 5)   # q, k, v, the bias and the offsets
    q, k, v = qkv(False)
    k.requires_grad_()
    call(delta, q, k, v).sum().backward()
    assert q.grad is None and v.grad is None and k.grad.shape == k.shape


@pytest.mark.parametrize("delta", [False, True])
def test_no_graph_without_need(delta):
    assert not call(delta, *qkv(False)).requires_grad
    with torch.no_grad():
        assert not call(delta, *qkv()).requires_grad
    with torch.inference_mode():
        assert call(delta, *qkv(False)).is_inference()


@pytest.mark.parametrize("delta", [False, True])
def test_what_is_refused(delta):
    with pytest.raises(NotImplementedError, match="mask is not differentiable"):
        call(delta, *qkv(), mask=plane(True))
    q, k, v = qkv()
    moved = q * 1
    out = call(delta, moved, k, v)
    moved.add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.sum().backward()
    q, k, v = qkv(False)
    with pytest.raises(RuntimeError):   # as an autograd function without a jvp / setup_context
        torch.func.grad(lambda q: call(delta, q, k, v).float().sum())(q)


def test_compiled_training_sees_both_operators():
    seen = []

    def backend(gm, inputs):
        seen.extend(str(n.target) for n in gm.graph.nodes)
        return gm

    from torch._dynamo.backends.common import aot_autograd
    leaves = qkv()
    torch._dynamo.reset()
    out = torch.compile(lambda q, k, v: call(False, q, k, v) * 2, backend=aot_autograd(fw_compiler=backend), fullgraph=True)(*leaves)
    torch.autograd.grad(out, leaves, torch.empty_like(out))
    assert "ops_rec.hstu_jagged.equal" in seen and "ops_rec.hstu_jagged_backward.equal" in seen
