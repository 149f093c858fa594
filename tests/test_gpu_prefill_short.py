"""GPU: short prompts of heads up to 128 columns go to the mma.sync kernel (64 rows and 64 keys per step): edges of its tiles, of the lengths and numbers of
blocks up to which it is taken, one buffer and two, packed rows with gaps that are cleared beside it; against float64, and no further from it than
the tcgen05 kernel."""
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


def rms(e):
    return float(e.double().pow(2).mean().sqrt())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,HQ,HKV,N,D", [(1, 1, 1, 1, 64), (2, 3, 1, 63, 128), (40, 8, 8, 64, 96), (1, 4, 2, 65, 64), (2, 5, 5, 127, 128), (1, 8, 2, 128, 40), (1, 4, 4, 129, 128),
                                          (3, 16, 4, 192, 128), (2, 4, 1, 193, 64), (1, 16, 2, 257, 120), (1, 2, 1, 384, 128)])
def test_dense(B, HQ, HKV, N, D, causal, dtype):
    q, k, v = draw(N + D, dtype, (B, HQ, N, D), (B, HKV, N, D), (B, HKV, N, D))
    run = lambda: dense(dtype)(q, k, v, causal)
    got, other = run(), by(2, run)
    assert torch.equal(got, by(1, run))
    want = torch.stack([exact(q[b], k[b], v[b], causal) for b in range(B)])
    assert (got - want).abs().max() < TOL[dtype]
    assert rms(got - want) < 1.02 * rms(other - want) + 1e-6


@pytest.mark.parametrize("B,HQ,N,D", [(1, 2, 385, 128), (2, 64, 193, 128), (64, 16, 65, 128), (8, 128, 129, 64)])
def test_longer_or_more_blocks_stay(B, HQ, N, D):
    """Past the lines (for a GPU of 148 SMs) the tcgen05 kernel's bits."""
    q, k, v = draw(N, torch.float16, (B, HQ, N, D), (B, HQ, N, D), (B, HQ, N, D))
    run = lambda: dense(torch.float16)(q, k, v, True)
    assert torch.equal(run(), by(2, run))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("lens,D", [([64, 1, 0, 17, 63], 128), ([128, 65, 3, 0, 192, 1], 64), ([192, 65, 3], 40), ([193, 1], 64), ([65, 2], 128)])
@pytest.mark.parametrize("causal", [True, False])
def test_packed_with_gaps(lens, D, causal, dtype):
    HQ, HKV, gap = 4, 2, 7
    cu = torch.tensor([gap] + lens).cumsum(0).to(torch.int32)
    total = int(cu[-1]) + gap
    q, k, v = draw(sum(lens), dtype, (total, HQ, D), (total, HKV, D), (total, HKV, D))
    for _ in range(20):
        junk = torch.full((total, HQ, D), 3.0, dtype=dtype, device="cuda")
        del junk                                                 # (the output's memory: rows that are not written would show)
        got = packed(dtype)(q, k, v, cu.cuda(), max(lens), causal)
    run = lambda: packed(dtype)(q, k, v, cu.cuda(), max(lens), causal)
    short = max(lens) <= (192 if D <= 64 else 64)
    assert torch.equal(got, by(1 if short else 2, run))
    assert not got[:gap].any() and not got[total - gap:].any()
    for a, e in zip(cu[:-1].tolist(), cu[1:].tolist()):
        if e > a:
            want = exact(q[a:e].transpose(0, 1), k[a:e].transpose(0, 1), v[a:e].transpose(0, 1), causal).transpose(0, 1)
            assert (got[a:e] - want).abs().max() < TOL[dtype]
