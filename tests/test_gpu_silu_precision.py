"""P and its gradient keep 32-bit accuracy up to their rounding to 16 bits wherever a call's head dims are not the 64 / 128 the
tensor-core kernels are tuned for: calls that isolate one score per output."""
import pytest
import torch

import ops_rec_b200

pytestmark = pytest.mark.gpu

op = ops_rec_b200.ascendc.attention.hstu_jagged
DIMS = [(32, 32), (8, 16), (64, 128), (128, 64), (96, 96)]
# one rounding to nearest of the result, and 2^-16 for the 32-bit arithmetic in front of it
BOUND = {torch.bfloat16: 2.0**-8 + 2.0**-16, torch.float16: 2.0**-11 + 2.0**-16}


def scores(dtype):
    return torch.linspace(-12, 8, 600, device="cuda").to(dtype)


def call(q, k, v, off, L):
    return op(q, k, v, None, None, 0, L, 1.0, off, None, None, 0, 1.0)


def first_column(x, dim):
    t = torch.zeros(len(x), 1, dim, device="cuda", dtype=x.dtype)
    t[:, 0, 0] = x
    return t


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("dqk,dv", DIMS)
@pytest.mark.parametrize("short", [True, False])
def test_forward(dtype, dqk, dv, short):
    """Row i scores x_i against every key and only key 0 has a value: out[i, 0] = silu(x_i).  As 600 sequences of one row
    (csrc/hstu_short.cu) and as one sequence of 600 (csrc/hstu_tc.cu)."""
    x = scores(dtype)
    n = len(x)
    off = torch.arange(n + 1, device="cuda") if short else torch.tensor([0, n], device="cuda")
    value = torch.ones_like(x) if short else torch.zeros_like(x).index_fill_(0, torch.zeros(1, dtype=torch.long, device="cuda"), 1)
    out = call(first_column(x, dqk), first_column(torch.ones_like(x), dqk), first_column(value, dv), off, n)
    want = torch.nn.functional.silu(x.double())
    assert ((out[:, 0, 0].double() - want).abs() <= BOUND[dtype] * want.abs()).all()
    assert (out[:, :, 1:] == 0).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("dqk,dv", DIMS)
def test_backward(dtype, dqk, dv):
    """Sequences of one row: dv = silu(x), dq = silu'(x), dk = silu'(x) x."""
    x = scores(dtype)
    off = torch.arange(len(x) + 1, device="cuda")
    leaves = [first_column(t, d).requires_grad_() for t, d in ((x, dqk), (torch.ones_like(x), dqk), (torch.ones_like(x), dv))]
    out = call(*leaves, off, 16)
    dq, dk, dvalue = (g[:, 0, 0].double() for g in torch.autograd.grad(out, leaves, first_column(torch.ones_like(x), dv)))
    xd = x.double().requires_grad_()
    silu = torch.nn.functional.silu(xd)
    slope, = torch.autograd.grad(silu.sum(), xd)
    bound = BOUND[dtype]
    assert ((dvalue - silu.detach()).abs() <= bound * silu.detach().abs()).all()
    # silu' passes through zero: 32-bit arithmetic on terms of size 1 there
    assert ((dq - slope).abs() <= bound * slope.abs() + 2.0**-20).all()
    assert ((dk - slope * x.double()).abs() <= 2.01 * bound * (slope * x.double()).abs() + 2.0**-17).all()
