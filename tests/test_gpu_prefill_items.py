"""GPU: the work items of a prefill belong to its launch alone, for each kernel that deals them out: a captured prefill replayed on one stream beside eager ones
on another, of different sizes and more items than SMs, gives the bits of each by itself, and so do calls by themselves afterwards."""
import pytest
import torch

pytestmark = pytest.mark.gpu
H, BF = torch.float16, torch.bfloat16


def rnd(*shape, dtype):
    return torch.randn(*shape, device="cuda").to(dtype)


def packed_call(D, lens):
    import flash_attn_v100 as fa
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    q, k, v = (rnd(sum(lens), h, D, dtype=H) for h in (8, 2, 2))
    return lambda: fa.forward_varlen_prefill_fp16(q, k, v, cu, max(lens), True)


def kv_call(lens):
    from flash_attn_v100_b200 import mixer_ops as mops
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    q, k, v = (rnd(sum(lens), h * 64, dtype=BF) for h in (8, 8, 8))
    slopes, st = torch.rand(8, device="cuda") * 0.1, torch.zeros(1, dtype=torch.int32, device="cuda")
    return lambda: mops.kv_prefill(q, k, v, cu, cu, max(lens), 8, 8, 0.125, slopes, st)


def latent_call(lens):
    from flash_attn_v100_b200 import hybrid_ops as hops
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    q, kv, kr = (rnd(sum(lens), c, dtype=BF) for c in (8 * 192, 8 * 256, 64))
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    return lambda: hops.latent_prefill(q, kv, kr, None, cu, cu, max(lens), 8, 128, 128, 0.07, st)


MANY, FEW = [700, 300, 1, 900] * 10, [300, 260, 129, 513] * 6        # sequences of different numbers of items, some of them empty
CALLS = {"up to 128 columns": lambda lens: packed_call(128, lens), "wide heads": lambda lens: packed_call(256, lens), "distance bias": kv_call, "latent": latent_call}


def wrong(got, want):
    return (got.view(torch.int16) != want.view(torch.int16)).any()


def fresh(call, like):
    """The call's result in memory that held something else."""
    junk = torch.full_like(like, float("nan"))
    del junk
    return call()


@pytest.mark.parametrize("kind", list(CALLS))
def test_replays_beside_eager_calls(kind):
    torch.manual_seed(1)
    many, few = CALLS[kind](MANY), CALLS[kind](FEW)
    want_many, want_few = many().clone(), few().clone()
    assert torch.isfinite(want_many).all() and torch.isfinite(want_few).all()
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=one):
        out = many()
    bad = torch.zeros(2, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    for _ in range(300):
        with torch.cuda.stream(one):
            out.fill_(float("nan"))
            graph.replay()
            bad[0] += wrong(out, want_many)
        with torch.cuda.stream(two):
            bad[1] += wrong(fresh(few, want_few), want_few)
    torch.cuda.synchronize()
    assert bad.tolist() == [0, 0]
    for _ in range(70):
        bad[1] += wrong(fresh(few, want_few), want_few)
    assert bad.tolist() == [0, 0]
