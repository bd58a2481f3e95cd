"""The backward's products on CTA pairs at the edges of their 256 x 256 tiles and 64-wide chunks, whole and split along the
contraction, against the oracle (checks and tolerances of test_in_linear_silu_bwd); and two calls give the same bits."""
import pytest
import torch

from tests.test_in_linear_silu_bwd import _case, _check, _run_cabi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n", [
    (1, 16, 64), (63, 16, 64), (257, 64, 256), (511, 80, 320),     # one tile or less; few chunks: whole products
    (1025, 16, 64), (4097, 48, 192), (8200, 64, 256),              # weight_grad split into parts, the last one shorter
    (200, 272, 4352), (129, 528, 2112),                            # x_grad split as well
    (2500, 256, 1024), (700, 1024, 4096)])                         # more tiles than half the pairs: not split
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_tile_edges_and_splits(m, k, n, dtype):
    c = _case(m, k, n, dtype, False, True, seed=m)
    got = _run_cabi(c)
    _check(c, got, f"{m} {k} {n}")
    for a, b in zip(got, _run_cabi(c)):
        assert (a is None and b is None) or torch.equal(a, b)
