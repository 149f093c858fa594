"""The projection-to-attention kernel gives the same bits in all its forms: one head per warp (few tokens) and four (many), whole
accesses and, at bases that are not aligned to them, element by element; head counts that four does not divide."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _call(dtype, qkv, qn, kn, cos, sin, table, cu, HQ, HKV, D, pages, shift=0):
    from flash_attn_v100_b200 import _lib
    lib = _lib.load()
    T, dev = qkv.size(0), qkv.device

    def place(*shape, like=None, dt=dtype):
        n = 1
        for s in shape:
            n *= s
        t = torch.zeros(n + shift, dtype=dt, device=dev)[shift:].view(*shape)
        if like is not None:
            t.copy_(like)
        return t
    q, k, v = place(T, HQ, D), place(T, HKV, D), place(T, HKV, D)
    kc, vc = place(pages, HKV, 16, D), place(pages, HKV, 16, D)
    x = place(*qkv.shape, like=qkv, dt=torch.bfloat16)
    entry = lib.fa_qkv_rope_append_f16 if dtype == torch.float16 else lib.fa_qkv_rope_append_bf16
    _lib.check(entry(x.data_ptr(), qn.data_ptr(), kn.data_ptr(), cos.data_ptr(), sin.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), kc.data_ptr(),
                     vc.data_ptr(), table.data_ptr(), None, cu.data_ptr(), T, cu.numel() - 1, HQ, HKV, D, 1e-6, pages, table.size(1),
                     torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return q, k, v, kc, vc


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("HQ,HKV,D", [(5, 1, 64), (32, 8, 128), (3, 3, 128), (2, 2, 256)])
def test_forms_agree(HQ, HKV, D, dtype):
    g = torch.Generator(device="cuda").manual_seed(D + HQ)
    lens = [1, 700, 16, 0, 983]
    T, per = sum(lens), 62
    qkv = torch.randn(T, (HQ + 2 * HKV) * D, generator=g, device="cuda").bfloat16()
    qn, kn = (torch.rand(D, generator=g, device="cuda").bfloat16() for _ in range(2))
    cos, sin = (torch.randn(T, D, generator=g, device="cuda") for _ in range(2))
    pages = len(lens) * per
    table = torch.randperm(pages, generator=g, device="cuda").to(torch.int32).view(len(lens), per)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    many = _call(dtype, qkv, qn, kn, cos, sin, table, cu, HQ, HKV, D, pages)
    odd = _call(dtype, qkv, qn, kn, cos, sin, table, cu, HQ, HKV, D, pages, shift=1)
    for a, b in zip(many, odd):
        assert torch.equal(a, b)
    at = 0
    for s, n in enumerate(lens):             # the first few tokens of every sequence in a call of their own: one head per warp
        if n == 0:
            continue
        m = min(n, 16)
        few = _call(dtype, qkv[at:at + m], qn, kn, cos[at:at + m], sin[at:at + m], table[s:s + 1].contiguous(), torch.tensor([0, m], dtype=torch.int32).cuda(),
                    HQ, HKV, D, pages)
        for a, b in zip(many[:3], few[:3]):
            assert torch.equal(a[at:at + m], b)
        page = table[s, 0]
        for a, b in zip(many[3:], few[3:]):
            assert torch.equal(a[page, :, :m], b[page, :, :m])
        at += n
