"""The forward kernel for batches of short sequences (csrc/hstu_short.cu) at the edges of its 64-key and 128-row tiles and of
the rule that sends calls to it, against the oracle (tolerances of the other parity tests)."""
import pytest
import torch

from oracle import hstu_paged_oracle as PO
from ops_rec_b200 import cabi
from tests._parity import assert_parity, run_cabi, to_cuda
from tests._util import make_case
from tests.test_paged import make_paged_case

pytestmark = pytest.mark.gpu

BF16, FP16 = torch.bfloat16, torch.float16


def run(args, short=True):
    """The call's output; it has to run on the kernel for short sequences (`short`), or on the other one."""
    cu = to_cuda(args)
    a, keep = cabi.make_args(cu["q"], cu["k"], cu["v"], None, cu["seq_offset"],
                             **{n: cu[n] for n in ("mask", "attn_bias", "mask_type", "max_seq_len", "max_seq_len_k",
                                                   "seq_offset_k", "num_context", "num_target", "target_group_size", "alpha")})
    assert cabi.kernel_kind(a) == 1 and cabi.short_form(a) == short
    return run_cabi(args)


@pytest.mark.parametrize("dims", [(64, 64), (8, 16), (48, 32)])
@pytest.mark.parametrize("L", [1, 15, 16, 17, 63, 64, 65, 127, 128, 129, 191, 192, 193, 257, 319])
@pytest.mark.parametrize("dtype,rab", [(BF16, None), (FP16, "batch"), (BF16, "shared3")])
def test_lengths(dims, L, dtype, rab):
    batch = 3 if L <= 160 else 48   # (a few longer sequences go to the other kernel)
    args = make_case(batch, 4, 2, *dims, L, L, dtype, seed=L, rab=rab, max_seq_len=(L + 7) // 8 * 8)
    out, status = run(args)
    assert status == 0
    assert_parity(out, args, label=f"{dims} {L}")


@pytest.mark.parametrize("dims", [(128, 128), (72, 80), (64, 128)])
@pytest.mark.parametrize("lo,hi,kw", [(1, 90, {}), (60, 95, dict(rab="shared3")), (1, 70, dict(mask_type=2)),
                                      (20, 60, dict(tgt=9, g=2, ctx=3, rab="batch", delta=True))])
def test_wide(dims, lo, hi, kw):
    args = make_case(7, 4, 2, *dims, lo, hi, BF16, seed=hi, max_seq_len=96, **kw)
    out, status = run(args)
    assert status == 0
    assert_parity(out, args, label=f"{dims} {hi}")


@pytest.mark.parametrize("rab,tgt", [(None, 5), ("shared3", 0)])
def test_many_items(rab, tgt):
    """More work items than eight per CTA: pairs of Q tiles, look-ups spread over the tiles before."""
    args = make_case(2600, 2, 2, 32, 32, 1, 150, BF16, seed=1, rab=rab, tgt=tgt, g=1 if tgt else 0, max_seq_len=160)
    out, status = run(args)
    assert status == 0
    assert_parity(out, args)


@pytest.mark.parametrize("batch,lo,hi,max_seq_len,short", [
    (24, 300, 339, None, False), (60, 280, 315, None, True), (300, 500, 1100, None, True), (10, 500, 1100, None, False),
    (20, 40, 80, 208, True), (20, 40, 80, 216, False), (120, 40, 80, 216, True), (120, 40, 80, 1024, False)])
def test_around_the_rule(batch, lo, hi, max_seq_len, short):
    """Both sides of the rule's lines give the oracle's result."""
    args = make_case(batch, 4, 4, 64, 64, lo, hi, BF16, seed=batch, max_seq_len=max_seq_len)
    out, status = run(args, short)
    assert status == 0
    assert_parity(out, args)


@pytest.mark.parametrize("poison", [float("nan"), float("inf")])
@pytest.mark.parametrize("D", [64, 128])
def test_neighbours_never_leak(poison, D):
    """Rows of the other sequences may hold anything."""
    args = make_case(5, 2, 2, D, D, 70, 90, BF16, seed=2)
    want, _ = run(args)
    off = args["seq_offset"].tolist()
    for n in ("q", "k", "v"):
        t = args[n].clone()
        t[:off[2]] = poison
        t[off[3]:] = poison
        args[n] = t
    out, status = run(args)
    assert status == 0
    assert torch.equal(out[off[2]:off[3]], want[off[2]:off[3]])


@pytest.mark.parametrize("page", [64, 128, 192, 256])
@pytest.mark.parametrize("D", [64, 32])
@pytest.mark.parametrize("hist,cand", [(63, 1), (64, 64), (65, 70), (130, 130)])
def test_paged_without_staging(page, D, hist, cand):
    """Pages read where they lie, targets from the call's own k / v: both segments' ends fall anywhere in a 64-key tile, and
    the unused rows of the cache hold NaNs."""
    args = make_paged_case(12, 4, 2, D, hist, cand, page, True, BF16, seed=hist + page)
    cache = args["kv_cache"].clone()
    used = torch.zeros(cache.shape[0], page, dtype=torch.bool)
    for b in range(len(args["last_page_len"])):
        ids = args["page_ids"][args["page_offsets"][b]:args["page_offsets"][b + 1]]
        for i, pid in enumerate(ids.tolist()):
            used[pid, :page if i + 1 < len(ids) else int(args["last_page_len"][b])] = True
    cache.transpose(1, 2)[~used] = float("nan")
    want = PO.hstu_paged_forward(**args, round_p=False, out_dtype=torch.float32)
    got, status = cabi.hstu_paged_forward(**{k: (v.cuda() if isinstance(v, torch.Tensor) else v)
                                             for k, v in dict(args, kv_cache=cache).items()}, return_status=True)
    assert status == 0
    torch.testing.assert_close(got.float().cpu(), want, rtol=1e-2, atol=1e-2)
    assert (got.float().cpu() - want).abs().max() <= 2e-2 * want.abs().max()
