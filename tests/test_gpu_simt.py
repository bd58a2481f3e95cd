"""The register-tiled CUDA-core kernels (fp32, and the 16-bit calls the tensor-core kernels leave) against the oracle, at
the edges of their 32-row / 64-key tiles and of their head dims; tolerances as in the other parity tests."""
import pytest
import torch

from ops_rec_b200 import cabi
from tests._parity import assert_parity, run_cabi
from tests._util import make_case
from tests.test_gpu_backward import assert_bwd_parity, make_bwd_case, run_bwd

pytestmark = pytest.mark.gpu

FP32, BF16, FP16 = torch.float32, torch.bfloat16, torch.float16


@pytest.mark.parametrize("dims", [(4, 16), (32, 32), (36, 48), (64, 64), (64, 128), (128, 64), (100, 112), (128, 128), (30, 32), (132, 32)])
@pytest.mark.parametrize("hi,delta,kw", [
    (1, False, {}), (33, False, dict(rab="batch")), (65, True, dict(ctx=3, tgt=7, g=2)),
    (130, False, dict(mask_type=2)), (129, True, dict(custom_mask=True, rab="shared3"))])
def test_forward(dims, hi, delta, kw):
    args = make_case(5, 4, 2, *dims, max(1, hi - 34), hi, FP32, seed=hi, delta=delta, **kw)
    out, status = run_cabi(args)
    assert status == 0
    assert_parity(out, args, label=f"{dims} {hi}")


@pytest.mark.parametrize("dims", [(4, 16), (32, 32), (36, 48), (64, 64), (64, 128), (100, 112), (128, 128), (30, 32)])
@pytest.mark.parametrize("maxl,dtype,kw", [
    (1, FP32, {}), (33, FP32, dict(bias=False)), (65, FP32, dict(ctx=3, tgt=7, g=2, delta=True)),
    (130, FP32, dict(mask_type=2, bias=False)), (97, FP32, dict(mask_type=3, delta=True)),
    (97, FP16, dict(mask_type=3)), (66, BF16, dict(mask_type=3, bias=False))])
def test_backward(dims, maxl, dtype, kw):
    grad, args = make_bwd_case(4, 4, 2, *dims, maxl, dtype, seed=maxl, **kw)
    got, status = run_bwd(grad, args)
    assert status == 0
    assert_bwd_parity(got, grad, args, label=f"{dims} {maxl}")


def test_misaligned_rows_take_the_other_kernel():
    """A query tensor that starts 4 bytes past a 16-byte boundary gives the same result (within rounding)."""
    args = make_case(3, 2, 2, 32, 32, 20, 90, FP32, seed=3)
    want, _ = run_cabi(args)
    flat = torch.empty(args["q"].numel() + 1, device="cuda")
    flat[1:] = args["q"].flatten().cuda()
    moved = dict(args, q=flat[1:].view(args["q"].shape))
    out, status = run_cabi(moved)
    assert status == 0
    torch.testing.assert_close(out, want, rtol=1e-5, atol=1e-6)


def test_quotient():
    """The quotient of the SiLU and the sigmoid is within half an ulp and 2^-17 of one of a / b for every b >= 1 (the bound
    beside the function), and the division's for infinities and NaN."""
    gen = torch.Generator(device="cuda").manual_seed(0)
    n = 1 << 22
    a = torch.randn(n, generator=gen, device="cuda") * torch.exp2(torch.rand(n, generator=gen, device="cuda") * 40 - 20)
    b = torch.exp2(torch.rand(n, generator=gen, device="cuda") * 127.99).clamp_(min=1)
    b[: n // 4] = 1 + torch.rand(n // 4, generator=gen, device="cuda")          # sigmoids of positive scores
    a[n // 8: n // 4] = 1
    a[n // 2: 3 * n // 4] = -torch.log(b[n // 2: 3 * n // 4] - 1).clamp_(min=-80, max=89)   # SiLU: x / (1 + exp(-x))
    got, want = cabi.debug_divide(a, b).double(), a.double() / b.double()
    ulp = torch.exp2(torch.floor(torch.log2(want.abs().clamp(min=2.0**-126))) - 23)
    normal = want.abs() >= 2.0**-126
    assert ((got - want).abs()[normal] <= (0.5 + 2.0**-17) * ulp[normal]).all()
    assert ((got - want).abs()[~normal] <= 2.0**-149).all()
    assert (got.float() != want.float()).float().mean() < 1e-5
    inf, nan = float("inf"), float("nan")
    x, y = (t.flatten().contiguous().cuda() for t in torch.meshgrid(
        torch.tensor([0.0, -0.0, 1.0, -88.0, inf, -inf, nan]), torch.tensor([1.0, 3.0, 2.0**127, inf, nan]), indexing="ij"))
    got, want = cabi.debug_divide(x, y), x / y
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.nan_to_num(9), want.nan_to_num(9))
