"""Prefill of wide heads (128 < D <= 256, `csrc/prefill_wide.cu`): edges of its 128-row and 128-key tiles, of the 64-key halves and of
the 64-column slabs, one item per CTA and many, against the fp32 oracle and the mma.sync kernel; its error against 64 bits; and which lengths
go to which kernel."""
import pytest
import torch

from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu

# P and V are fp16 (relative rounding 2^-11 each, averaging out over the keys), the output is rounded once more: the bound of the other
# fp16 prefill tests
TOL = 2e-3


@pytest.fixture
def fa():
    """The module with the tcgen05 kernels required, so that nothing here can pass on the other kernel."""
    import flash_attn_v100
    from flash_attn_v100_b200 import ops
    ops.set_prefill_impl(2)
    yield flash_attn_v100
    ops.set_prefill_impl(0)


def _by(impl, fn):
    from flash_attn_v100_b200 import ops
    ops.set_prefill_impl(impl)
    try:
        return fn()
    finally:
        ops.set_prefill_impl(2)


def _dense(B, HQ, HKV, N, D, seed):
    g = torch.Generator().manual_seed(seed)
    return [torch.randn(B, h, N, D, generator=g).half() for h in (HQ, HKV, HKV)]


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,HQ,HKV,N,D", [(1, 1, 1, 1, 256), (1, 2, 1, 63, 136), (2, 3, 1, 64, 192), (1, 4, 2, 65, 200), (1, 2, 2, 127, 256), (1, 2, 1, 128, 248),
                                          (1, 5, 5, 129, 160), (1, 2, 1, 257, 256), (1, 2, 1, 700, 256), (3, 16, 4, 900, 256)])
def test_dense_against_oracle(fa, B, HQ, HKV, N, D, causal):
    q, k, v = _dense(B, HQ, HKV, N, D, N * D)
    got = fa.forward_prefill_gqa_fp16(q.cuda(), k.cuda(), v.cuda(), causal).float().cpu()
    kk, vv = (t.float().repeat_interleave(HQ // HKV, 1) for t in (k, v))
    s = q.float() @ kk.transpose(-1, -2) * D ** -0.5
    if causal:
        s = s.masked_fill(torch.ones(N, N).triu(1).bool(), float("-inf"))
    assert (got - torch.softmax(s, -1) @ vv).abs().max() < TOL


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("D", [256, 168])
def test_packed_against_oracle_and_other_kernel(fa, causal, D):
    from flash_attn_v100_b200 import ops
    lens = [1, 130, 0, 64, 385, 5, 1111]
    cu = torch.tensor([3] + lens).cumsum(0).to(torch.int32)        # rows before the first and behind the last sequence
    total, HQ, HKV = int(cu[-1]) + 9, 8, 2
    g = torch.Generator().manual_seed(D)
    q, k, v = (torch.randn(total, h, D, generator=g).half() for h in (HQ, HKV, HKV))
    args = (q.cuda(), k.cuda(), v.cuda(), cu.cuda(), max(lens), causal)
    got = fa.forward_varlen_prefill_fp16(*args)
    bf = fa.forward_varlen_prefill_fp16(*args, out_dtype=torch.bfloat16)
    other = _by(1, lambda: fa.forward_varlen_prefill_fp16(*args))
    a, e = int(cu[0]), int(cu[-1])
    assert not got[:a].any() and not got[e:].any()
    ref = orc.varlen_prefill(q[a:e], k[a:e], v[a:e], cu - a, causal, final_cast=False)
    assert (got[a:e].float().cpu() - ref).abs().max() < TOL
    assert (got.float() - other.float()).abs().max() < TOL
    assert ((bf.float() - got.float()).abs() <= 2 ** -8 * got.float().abs() + 1e-6).all()      # one more rounding, to bfloat16
    ops.check_prefill_errors()


def test_neighbours_that_are_not_numbers(fa):
    """Keys and values of other sequences never reach a result, whatever they hold."""
    lens, D = [70, 200, 33], 256
    cu = torch.tensor([0, 70, 270, 303], dtype=torch.int32)
    g = torch.Generator().manual_seed(5)
    q, k, v = (torch.randn(303, 2, D, generator=g).half() for _ in range(3))
    want = fa.forward_varlen_prefill_fp16(q.cuda(), k.cuda(), v.cuda(), cu.cuda(), max(lens), True)
    k[70:270] = float("nan")
    v[70:270] = float("inf")
    got = fa.forward_varlen_prefill_fp16(q.cuda(), k.cuda(), v.cuda(), cu.cuda(), max(lens), True)
    assert torch.equal(got[:70], want[:70]) and torch.equal(got[270:], want[270:])


def test_growing_scores(fa):
    """Row maxima that keep growing by far more than the rescale threshold, and a row whose late keys dwarf the early ones."""
    q, k, v = _dense(1, 2, 1, 640, 256, 11)
    k = k * torch.linspace(0.1, 6, 640)[None, None, :, None].half()
    got = fa.forward_prefill_gqa_fp16(q.cuda(), k.cuda(), v.cuda(), True).float().cpu()
    s = q.float() @ k.float().repeat_interleave(2, 1).transpose(-1, -2) / 16
    s = s.masked_fill(torch.ones(640, 640).triu(1).bool(), float("-inf"))
    assert (got - torch.softmax(s, -1) @ v.float().repeat_interleave(2, 1)).abs().max() < TOL * 2   # values stand out up to 5: twice the rounding


def _error(got, q, k, v, causal):
    """Relative 2-norm against 64 bits."""
    r, n = q.size(1) // k.size(1), q.size(2)
    k, v = (t.double().repeat_interleave(r, 1) for t in (k, v))
    s = q.double() @ k.transpose(-1, -2) * q.size(3) ** -0.5
    if causal:
        s = s.masked_fill(torch.ones(n, n, device=q.device).triu(1).bool(), float("-inf"))
    ref = torch.softmax(s, -1) @ v
    return ((got.double() - ref).norm() / ref.norm()).item()


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("N,D,spread", [(130, 256, 1.0), (1000, 192, 1.0), (2048, 256, 1.0), (2048, 136, 3.0), (700, 256, 0.3)])
def test_error_no_larger_than_the_other_kernels(fa, N, D, spread, causal):
    """The reference exponent of a row lags behind its maximum here, so the largest weight is not exactly 1, as it is in the mma.sync kernel; what
    the rounding to fp16 leaves of the weights has to make up for that, for flat scores and for peaked ones."""
    q, k, v = (t.cuda() for t in _dense(2, 4, 2, N, D, N))
    q = (q.float() * spread).half()
    run = lambda: fa.forward_prefill_gqa_fp16(q, k, v, causal)
    assert _error(run(), q, k, v, causal) <= _error(_by(1, run), q, k, v, causal)


@pytest.mark.parametrize("B,HQ,N,wide", [(1, 2, 64, False), (1, 2, 128, False), (1, 2, 129, True), (2, 64, 64, False), (2, 64, 65, True), (3, 100, 16, False)])
def test_short_prompts_stay_with_the_other_kernel(fa, B, HQ, N, wide):
    """Which kernel a length goes to shows in the bits: the rounding of the two differs in some element of every such output."""
    q, k, v = (t.cuda() for t in _dense(B, HQ, HQ // 2, N, 256, N + HQ))
    run = lambda: fa.forward_prefill_gqa_fp16(q, k, v, True)
    mma, tc = _by(1, run), run()
    assert not torch.equal(mma, tc)
    assert torch.equal(_by(0, run), tc if wide else mma)
