"""GPU: short prompts of heads up to 128 columns, at the edges of both kernels' tiles, dense and packed between gaps, against float64; and a sequence's bits, which are the
same in every call that it comes in."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# weights and outputs have 11 (8) bits: the bound of the other prefill tests, and eight times that for bfloat16
TOL = {torch.float16: 2e-3, torch.bfloat16: 1.6e-2}


def exact(q, k, v, causal):
    """[H, N, D] in float64"""
    k, v = (t.double().repeat_interleave(q.size(0) // t.size(0), 0) for t in (k, v))
    s = q.double() @ k.transpose(-1, -2) * q.size(-1) ** -0.5
    if causal:
        s = s.masked_fill(torch.ones(s.shape[-2:], dtype=torch.bool, device=s.device).triu(1), float("-inf"))
    return torch.softmax(s, -1) @ v


def by(impl, fn):
    from flash_attn_v100_b200 import ops
    ops.set_prefill_impl(impl)
    try:
        return fn()
    finally:
        ops.set_prefill_impl(0)


def draw(seed, dtype, *shapes):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(*s, generator=g, device="cuda").to(dtype) for s in shapes]


def dense(dtype):
    import flash_attn_v100 as fa
    from flash_attn_v100_b200 import ops
    return fa.forward_prefill_gqa_fp16 if dtype == torch.float16 else ops.forward_prefill_gqa_bf16


def packed(dtype):
    import flash_attn_v100 as fa
    from flash_attn_v100_b200 import ops
    return fa.forward_varlen_prefill_fp16 if dtype == torch.float16 else ops.forward_varlen_prefill_bf16


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,HQ,HKV,N,D", [(1, 1, 1, 1, 64), (2, 3, 1, 63, 128), (40, 8, 8, 64, 96), (1, 4, 2, 65, 64), (2, 5, 5, 127, 128), (1, 8, 2, 128, 40), (1, 4, 4, 129, 128),
                                          (3, 16, 4, 192, 128), (2, 4, 1, 193, 64), (1, 16, 2, 257, 120), (1, 2, 1, 384, 128)])
def test_dense(B, HQ, HKV, N, D, causal, dtype):
    q, k, v = draw(N + D, dtype, (B, HQ, N, D), (B, HKV, N, D), (B, HKV, N, D))
    want = torch.stack([exact(q[b], k[b], v[b], causal) for b in range(B)])
    for impl in (1, 2, 3):
        assert (by(impl, lambda: dense(dtype)(q, k, v, causal)) - want).abs().max() < TOL[dtype], impl


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("lens,D", [([64, 1, 0, 17, 63], 128), ([128, 65, 3, 0, 192, 1], 64), ([192, 65, 3], 40), ([193, 1], 64), ([65, 2], 128), ([700, 64, 65, 200], 128)])
@pytest.mark.parametrize("causal", [True, False])
def test_packed_with_gaps(lens, D, causal, dtype):
    HQ, HKV, gap = 4, 2, 7
    cu = torch.tensor([gap] + lens).cumsum(0).to(torch.int32)
    total = int(cu[-1]) + gap
    q, k, v = draw(sum(lens), dtype, (total, HQ, D), (total, HKV, D), (total, HKV, D))
    for impl in (0, 1, 3):
        for _ in range(20):
            junk = torch.full((total, HQ, D), 3.0, dtype=dtype, device="cuda")
            del junk                                             # (the output's memory: rows that are not written would show)
            got = by(impl, lambda: packed(dtype)(q, k, v, cu.cuda(), max(lens), causal))
        assert not got[:gap].any() and not got[total - gap:].any()
        for a, e in zip(cu[:-1].tolist(), cu[1:].tolist()):
            if e > a:
                want = exact(q[a:e].transpose(0, 1), k[a:e].transpose(0, 1), v[a:e].transpose(0, 1), causal).transpose(0, 1)
                assert (got[a:e] - want).abs().max() < TOL[dtype]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [40, 64, 96, 128])
@pytest.mark.parametrize("HQ,HKV,causal", [(4, 2, True), (3, 1, True), (4, 2, False)])
def test_bits_do_not_depend_on_the_call(HQ, HKV, causal, D, dtype):
    """A sequence beside longer and shorter ones, alone, behind a larger bound and in dense batches."""
    lens = [50, 500, 64, 1, 65, 150, 192, 193, 300]
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32)
    q, k, v = draw(D, dtype, *((sum(lens), h, D) for h in (HQ, HKV, HKV)))
    together = packed(dtype)(q, k, v, cu.cuda(), max(lens), causal)
    for a, n in zip(cu.tolist(), lens):
        part = [t[a:a + n].contiguous() for t in (q, k, v)]
        one = torch.tensor([0, n], dtype=torch.int32, device="cuda")
        for bound in (n, 1000):
            assert torch.equal(packed(dtype)(*part, one, bound, causal), together[a:a + n]), (n, bound)
        for B in (1, 200):
            whole = [t.transpose(0, 1)[None].expand(B, -1, -1, -1).contiguous() for t in part]
            assert torch.equal(dense(dtype)(*whole, causal), together[a:a + n].transpose(0, 1)[None].expand(B, -1, -1, -1)), (n, B)
