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


def _clear(out, cu, longest):
    from flash_attn_v100_b200 import _lib
    lib = _lib.load()
    _lib.check(lib.fa_prefill_varlen_clear(out.data_ptr(), cu.data_ptr(), cu.numel() - 1, out.size(0), longest, out.size(1), torch.cuda.current_stream().cuda_stream))


# (2000003 rows of 16 bytes: a block's share is more than it marks at a time)
@pytest.mark.parametrize("rows,row_bytes", [(1, 16), (1000, 8192), (40000, 8192), (2000003, 16), (33, 512), (5000, 528)])
@pytest.mark.parametrize("offsets", ["few", "many", "out of order"])
def test_clear_touches_nothing_else(rows, row_bytes, offsets):
    cu = [rows // 10, rows // 3, rows // 3, rows // 2]
    if offsets == "many":
        cu = sorted((torch.rand(700, generator=torch.Generator().manual_seed(rows)) * rows).int().tolist())
    elif offsets == "out of order":
        cu = [rows // 3, rows // 10, rows // 2, rows // 4]
    longest = max(1, rows // 8 if offsets != "many" else rows // 700)
    memory = torch.ones(rows + 2, row_bytes, dtype=torch.uint8, device="cuda")       # a row on either side that must stay
    out = memory[1:-1]
    _clear(out, torch.tensor(cu, dtype=torch.int32, device="cuda"), longest)
    gap, covered = torch.zeros(rows, dtype=torch.bool), torch.zeros(rows, dtype=torch.bool)
    gap[:cu[0]] = gap[cu[-1]:] = True
    for a, e in zip(cu, cu[1:]):
        covered[a:min(e, a + longest)] = True
        gap[a + longest:e] = True
    assert bool((gap | covered).all())                       # what no sequence covers lies in a gap
    rows_of = memory.cpu().view(rows + 2, row_bytes)
    assert bool(rows_of[0].all()) and bool(rows_of[-1].all())
    assert torch.equal(rows_of[1:-1], (~gap).to(torch.uint8)[:, None].expand(rows, row_bytes))


@pytest.mark.parametrize("batch", [1, 64, 300, 2000])
def test_long_gap_at_the_rate_of_a_fill(batch):
    """A buffer padded to a fixed size: the gap behind the sequences is nearly all of it.  A fill is the time it took before there was
    a clear; the line is four of them, and the clear by few blocks took up to 60."""
    rows, row_bytes = 65536, 8192
    out = torch.ones(rows, row_bytes, dtype=torch.uint8, device="cuda")
    cu = torch.arange(batch + 1, dtype=torch.int32, device="cuda")

    def fastest(fn):
        times = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            fn()
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)
    assert fastest(lambda: _clear(out, cu, 1)) < 4 * fastest(out.zero_)


@pytest.mark.parametrize("D,longest", [(128, 1000), (64, 30), (128, 64), (256, 1000), (256, 20)])
def test_no_sequence_has_rows(D, longest):
    """All sequences empty, the whole of a large output to be cleared: nothing that follows on the stream sees it before, although no block of the attention
    has anything to store."""
    from flash_attn_v100_b200 import ops
    total, H = 16384, 32768 // D
    q, k, v = (torch.randn(total, h, D, dtype=torch.float16, device="cuda") for h in (H, 1, 1))
    cu = torch.full((4,), 7, dtype=torch.int32, device="cuda")
    run = lambda: ops.forward_varlen_prefill_fp16(q, k, v, cu, longest, True)
    run()
    for _ in range(5):
        stale = torch.full((total, H, D), float("nan"), dtype=torch.float16, device="cuda")
        del stale
        torch.cuda._sleep(1000000)                     # everything below is in the queue by the time it starts
        got = run()
        rows = got[1023::1024].clone()
        assert not rows.any() and not got.any()
        del got


@pytest.mark.parametrize("D", [64, 128, 200])
@pytest.mark.parametrize("cu,longest", [([60, 100, 20], 1000), ([60, 500, 20, 55], 300), ([60, 90, 500, 20], 1000), ([-5, 30, 90, 400], 1000), ([-5, 30, 90], 40), ([590, 700], 300)])
def test_offsets_out_of_order_or_range(cu, longest, D):
    """Rows that a sequence covers are its result although they lie in another one's gap, too; all others are zeros; a sequence that starts below 0 has no rows."""
    from flash_attn_v100_b200 import ops
    total, H = 600, 4
    q, k, v = (torch.randn(total, h, D, dtype=torch.float16, device="cuda") for h in (H, 2, 2))
    call = lambda t, cu: ops.forward_varlen_prefill_fp16(*t, torch.tensor(cu, dtype=torch.int32, device="cuda"), longest, True)
    want = torch.zeros(total, H, D, dtype=torch.float16, device="cuda")
    for a, e in zip(cu, cu[1:]):
        n = min(e, total, a + longest) - a
        if a >= 0 and n > 0:
            want[a:a + n] = call([t[a:a + n].contiguous() for t in (q, k, v)], [0, n])
    for _ in range(10):
        stale = torch.full((total, H, D), float("nan"), dtype=torch.float16, device="cuda")
        del stale
        assert torch.equal(call((q, k, v), cu), want)
