"""Decode where a segment is cut into equal parts, one per CTA, and the neighbouring cases where it is not (more segments than CTAs, long
sequences): lengths at the edges of pages, of what a CTA's rings hold and of the parts; every operator against plain attention."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(q, k, v):
    """q [HQ, D], k, v [HKV, n, D] in fp64 -> [HQ, D]"""
    hq, d = q.shape
    hkv = k.size(0)
    q = q.double().view(hkv, hq // hkv, d)
    return (torch.softmax(q @ k.double().transpose(1, 2) * d ** -0.5, -1) @ v.double()).view(hq, d)


LENS = [[1], [16, 17, 0, 128, 129], [127, 128, 130, 143, 144, 145, 256, 257], [1000, 1024, 999, 1023], [5000], [8, 4096, 33], [64] * 300, [0, 0]]


@pytest.mark.parametrize("HQ,HKV,D", [(32, 8, 128), (4, 1, 64), (17, 1, 128), (40, 2, 256), (6, 3, 96)])
@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_paged(lens, HQ, HKV, D, dtype):
    from flash_attn_v100_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + D)
    B, need = len(lens), [(n + 15) // 16 for n in lens]
    count, width = max(1, sum(need)), max(1, max(need))
    k, v = (torch.randn(count, HKV, 16, D, generator=g, device="cuda").to(dtype) for _ in range(2))
    q = torch.randn(B, HQ, 1, D, generator=g, device="cuda").to(dtype)
    perm, table, at = torch.randperm(count, generator=g, device="cuda").to(torch.int32), torch.zeros(B, width, dtype=torch.int32, device="cuda"), 0
    for b, n in enumerate(need):
        table[b, :n] = perm[at:at + n]
        at += n
    fn = ops.forward_paged_decode_gqa_fp16 if dtype == torch.float16 else ops.forward_paged_decode_gqa_bf16
    out = [fn(q, k, v, table, torch.tensor(lens, dtype=torch.int32, device="cuda"), width) for _ in range(2)]
    ops.check_async_errors()
    assert torch.equal(out[0], out[1])                   # the arrival counters are back at zero
    # P and the result are rounded to 2^-11 or 2^-8, values stand out up to 4 where few keys are seen
    tol = 2e-3 if dtype == torch.float16 else 1.6e-2
    for b in sorted({0, B // 2, B - 1}):
        n = lens[b]
        got = out[0][b, :, 0].double()
        if n == 0:
            assert not got.any()
            continue
        ids = table[b, :need[b]].long()
        ref = _ref(q[b, :, 0], *(t[ids].transpose(0, 1).reshape(HKV, -1, D)[:, :n] for t in (k, v)))
        assert ((got - ref).abs() <= tol + ref.abs() * tol / 4).all()


@pytest.mark.parametrize("B,N,used", [(1, 200, 129), (3, 3000, 2999), (40, 90, 77), (2, 700, 513)])
def test_contiguous_operators(B, N, used):
    from flash_attn_v100_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(N)
    HQ, HKV, D = 16, 4, 128
    q, k, v = (torch.randn(B, h, n, D, generator=g, device="cuda").half() for h, n in ((HQ, 1), (HKV, N), (HKV, N)))
    b = B - 1
    dense = _ref(q[b, :, 0], k[b, :, :used], v[b, :, :used])
    close = lambda got, ref, tol: bool(((got[b, :, 0].double() - ref).abs() <= tol + ref.abs() * tol / 4).all())
    assert close(ops.forward_decode_gqa_fp16(q, k, v, True, used - 1), dense, 2e-3)
    last = torch.full((B,), used - 1, dtype=torch.int32, device="cuda")
    assert close(ops.forward_continuous_batching_fp16(q, k, v, last, True), dense, 2e-3)
    window, sink = used // 2, 5
    seen = (torch.arange(used) < sink) | (torch.arange(used) >= used - window)
    assert close(ops.forward_decode_sliding_window_gqa(q, k, v, True, used - 1, window, sink),
                 _ref(q[b, :, 0], k[b, :, :used][:, seen.cuda()], v[b, :, :used][:, seen.cuda()]), 2e-3)
    k8, v8 = (torch.randint(-127, 128, (B, HKV, N, D), generator=g, device="cuda").to(torch.int8) for _ in range(2))
    ks, vs = ((torch.rand(B, HKV, N, generator=g, device="cuda") * 0.01 + 0.02).half() for _ in range(2))
    got = ops.forward_decode_int8_kv_cache_gqa(q, k8, v8, ks, vs, used - 1)
    assert close(got, _ref(q[b, :, 0], k8[b, :, :used].double() * ks[b, :, :used, None].double(), v8[b, :, :used].double() * vs[b, :, :used, None].double()), 3e-3)
    qs, kq = (q.abs().amax(-1).float().squeeze(-1) / 127).contiguous(), (k.abs().amax(-1).float() / 127).contiguous()
    whole = lambda x, s: (lambda y: (y.sign() * (y.abs() + 0.5).floor()).clamp(-127, 127))((x.float() / s.float()).double())
    got = ops.forward_decode_int8_gqa(q, k, v, qs, kq, used - 1)
    ref = _ref(whole(q[b, :, 0], qs[b][:, None]) * qs[b][:, None].double(), whole(k[b, :, :used], kq[b, :, :used, None]) * kq[b, :, :used, None].double(), v[b, :, :used])
    assert close(got, ref, 2e-3)
    ops.check_async_errors()
