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


@pytest.mark.parametrize("HQ,HKV,D", [(32, 8, 128), (4, 1, 64), (17, 1, 128), (40, 2, 256), (6, 3, 96), (3, 1, 136)])
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
    for b in range(B) if B < 100 else (0, B // 2, B - 1):
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
    last = torch.full((B,), used - 1, dtype=torch.int32, device="cuda")
    window, sink = used // 2, 5
    seen = ((torch.arange(used) < sink) | (torch.arange(used) >= used - window)).cuda()
    k8, v8 = (torch.randint(-127, 128, (B, HKV, N, D), generator=g, device="cuda").to(torch.int8) for _ in range(2))
    ks, vs = ((torch.rand(B, HKV, N, generator=g, device="cuda") * 0.01 + 0.02).half() for _ in range(2))
    qs, kq = (q.abs().amax(-1).float().squeeze(-1) / 127).contiguous(), (k.abs().amax(-1).float() / 127).contiguous()
    whole = lambda x, s: (lambda y: (y.sign() * (y.abs() + 0.5).floor()).clamp(-127, 127))((x.float() / s.float()).double())
    got = [ops.forward_decode_gqa_fp16(q, k, v, True, used - 1), ops.forward_continuous_batching_fp16(q, k, v, last, True),
           ops.forward_decode_sliding_window_gqa(q, k, v, True, used - 1, window, sink),
           ops.forward_decode_int8_kv_cache_gqa(q, k8, v8, ks, vs, used - 1), ops.forward_decode_int8_gqa(q, k, v, qs, kq, used - 1)]
    for b in sorted({0, B - 1}):
        x, kb, vb = q[b, :, 0], k[b, :, :used], v[b, :, :used]
        dense = _ref(x, kb, vb)
        refs = [dense, dense, _ref(x, kb[:, seen], vb[:, seen]),
                _ref(x, k8[b, :, :used].double() * ks[b, :, :used, None].double(), v8[b, :, :used].double() * vs[b, :, :used, None].double()),
                _ref(whole(x, qs[b][:, None]) * qs[b][:, None].double(), whole(kb, kq[b, :, :used, None]) * kq[b, :, :used, None].double(), vb)]
        for o, ref, tol in zip(got, refs, (2e-3, 2e-3, 2e-3, 3e-3, 2e-3)):
            assert ((o[b, :, 0].double() - ref).abs() <= tol + ref.abs() * tol / 4).all()
    ops.check_async_errors()


@pytest.mark.parametrize("width", [40, 2000])
def test_captured_decode_whose_lengths_grow(width):
    """A decode captured once and replayed while its sequences grow, as a generation loop has it: the CTAs per segment follow from the width
    of the table, what each of them does from the lengths on the device, from one part to several and back.  `width` 40: equal parts; 2000: the even cut."""
    from flash_attn_v100_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(width)
    B, HQ, HKV, D, most = 3, 8, 2, 128, 640
    pages = B * (most // 16)
    k, v = (torch.randn(pages, HKV, 16, D, generator=g, device="cuda").half() for _ in range(2))
    q = torch.randn(B, HQ, 1, D, generator=g, device="cuda").half()
    table = torch.zeros(B, width, dtype=torch.int32, device="cuda")
    table[:, :most // 16] = torch.randperm(pages, generator=g, device="cuda").to(torch.int32).view(B, -1)
    lens = torch.tensor([1, 17, 100], dtype=torch.int32, device="cuda")
    run = lambda: ops.forward_paged_decode_gqa_fp16(q, k, v, table, lens, width)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        run()
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = run()
    for now in ([1, 17, 100], [128, 129, 0], [129, 255, 640], [640, 513, 300], [2, 640, 16]):
        lens.copy_(torch.tensor(now, dtype=torch.int32))
        graph.replay()
        eager = run()
        assert torch.equal(out, eager)
        for b, n in enumerate(now):
            if n == 0:
                assert not out[b].any()
                continue
            ids = table[b, :(n + 15) // 16].long()
            ref = _ref(q[b, :, 0], *(t[ids].transpose(0, 1).reshape(HKV, -1, D)[:, :n] for t in (k, v)))
            assert ((out[b, :, 0].double() - ref).abs() <= 2e-3 + ref.abs() * 5e-4).all()
    ops.check_async_errors()
