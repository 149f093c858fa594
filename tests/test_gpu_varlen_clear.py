"""Rows of a packed output that no sequence covers are zeros, whatever the memory held before: gaps before, between (sequences longer than
max_seqlen) and behind the sequences, for each of the prefill kernels."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,dtype", [(128, torch.float16), (64, torch.bfloat16), (96, torch.float16), (200, torch.float16)])
@pytest.mark.parametrize("cu,behind,longest", [([0, 5, 5, 300], 0, 295), ([7, 100, 101], 1, 1000), ([0, 400, 410, 1000], 33, 256), ([0] * 301 + [2], 5000, 2)])
def test_uncovered_rows_are_zero(D, dtype, cu, behind, longest):
    from flash_attn_v100_b200 import ops
    total, HQ, HKV = cu[-1] + behind, 4, 2
    q, k, v = (torch.randn(total, h, D, dtype=dtype, device="cuda") for h in (HQ, HKV, HKV))
    fn = ops.forward_varlen_prefill_fp16 if dtype == torch.float16 else ops.forward_varlen_prefill_bf16
    covered = torch.zeros(total, dtype=torch.bool)
    for a, e in zip(cu, cu[1:]):
        covered[a:min(e, a + longest)] = True
    for _ in range(2):
        stale = torch.full((total, HQ, D), float("nan"), dtype=dtype, device="cuda")      # the next allocation of that size gets this memory
        del stale
        got = fn(q, k, v, torch.tensor(cu, dtype=torch.int32, device="cuda"), longest, True)
        assert not got[~covered.cuda()].any()
        assert bool((got[covered.cuda()] != 0).any(-1).all()) and not got.isnan().any()
        del got


@pytest.mark.parametrize("rows,row_bytes", [(1, 16), (1000, 8192), (40000, 8192)])
def test_clear_touches_nothing_else(rows, row_bytes):
    from flash_attn_v100_b200 import _lib
    lib = _lib.load()
    out = torch.ones(rows, row_bytes, dtype=torch.uint8, device="cuda")
    cu = [rows // 10, rows // 3, rows // 3, rows // 2]
    longest = max(1, rows // 8)
    _lib.check(lib.fa_prefill_varlen_clear(out.data_ptr(), torch.tensor(cu, dtype=torch.int32, device="cuda").data_ptr(), 3, rows, longest, row_bytes,
                                           torch.cuda.current_stream().cuda_stream))
    want = torch.zeros(rows, dtype=torch.uint8)
    for a, e in zip(cu, cu[1:]):
        want[a:min(e, a + longest)] = 1
    assert torch.equal(out.cpu(), want[:, None].expand(rows, row_bytes))
