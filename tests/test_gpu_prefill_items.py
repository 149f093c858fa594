"""GPU: the work items of a prefill belong to its launch alone, for each kernel that deals them out: a captured prefill replayed on one stream beside eager ones
on another, of different sizes and more items than SMs, gives the bits of each by itself, and so do calls by themselves afterwards.  Long and short sequences in
one call, whose items are found by walking them."""
import pytest
import torch

pytestmark = pytest.mark.gpu
H, BF = torch.float16, torch.bfloat16


def rnd(*shape, dtype):
    return torch.randn(*shape, device="cuda").to(dtype)


def offsets(lens):
    return torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()


def packed(D):
    import flash_attn_v100 as fa
    return lambda T: [rnd(T, h, D, dtype=H) for h in (8, 2, 2)], lambda t, cu, longest: fa.forward_varlen_prefill_fp16(*t, cu, longest, True)


def biased():
    from flash_attn_v100_b200 import mixer_ops as mops
    slopes, st = torch.linspace(0.01, 0.1, 8, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    return lambda T: [rnd(T, h * 64, dtype=BF) for h in (8, 8, 8)], lambda t, cu, longest: mops.kv_prefill(*t, cu, cu, longest, 8, 8, 0.125, slopes, st)


def latent():
    from flash_attn_v100_b200 import hybrid_ops as hops
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    return (lambda T: [rnd(T, c, dtype=BF) for c in (8 * 192, 8 * 256, 64)],
            lambda t, cu, longest: hops.latent_prefill(*t, None, cu, cu, longest, 8, 128, 128, 0.07, st))


# name -> (tensors of that many tokens, the call with them, offsets and a bound on the lengths)
KINDS = {"up to 128 columns": lambda: packed(128), "wide heads": lambda: packed(256), "distance bias": biased, "latent": latent}


def call_of(kind, lens):
    make, run = KINDS[kind]()
    tensors, cu = make(sum(lens)), offsets(lens)
    return lambda: run(tensors, cu, max(lens))


MANY, FEW = [700, 300, 1, 900] * 10, [300, 260, 129, 513] * 6        # sequences of different numbers of items


def wrong(got, want):
    return (got.view(torch.int16) != want.view(torch.int16)).any()


def fresh(call, like):
    """The call's result in memory that held something else."""
    junk = torch.full_like(like, float("nan"))
    del junk
    return call()


@pytest.mark.parametrize("kind", list(KINDS))
def test_replays_beside_eager_calls(kind):
    torch.manual_seed(1)
    many, few = call_of(kind, MANY), call_of(kind, FEW)
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


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("lens", [[3000] + [30, 1, 0, 300] * 30, [5] * 40 + [2000, 0, 0] + [700] * 3 + [65] * 70, [0] * 70 + [1000] + [0] * 5, [129] * 33])
def test_long_and_short_sequences(kind, lens):
    """Items are found among 32 sequences at a time, level by level: every sequence gives the bits of itself alone (with a distance bias not quite: the rows of the next
    sequence that share a tile have a say in how its sums are scaled)."""
    torch.manual_seed(2)
    make, run = KINDS[kind]()
    tensors, cu = make(sum(lens)), torch.tensor([0] + lens).cumsum(0).tolist()
    whole = run(tensors, offsets(lens), max(lens))
    for n in sorted(set(lens) - {0}):
        alone = None
        for i, m in enumerate(lens):
            if m == n:
                part = [t[cu[i]:cu[i] + n].contiguous() for t in tensors]
                alone = run(part, offsets([n]), max(lens))
                got = whole[cu[i]:cu[i] + n]
                assert (got - alone).abs().max() < 2 ** -4 if kind == "distance bias" else not wrong(got, alone), (n, i)


@pytest.mark.parametrize("D", [128, 256])
def test_more_items_than_rows_allow(D):
    """Offsets out of order, the same rows again and again: more items than sequences without common rows can have."""
    import flash_attn_v100 as fa
    n, times = 700, 40
    q, k, v = (rnd(n, h, D, dtype=H) for h in (32, 8, 8))
    i32 = lambda *x: torch.tensor(x, dtype=torch.int32, device="cuda")
    one = fa.forward_varlen_prefill_fp16(q, k, v, i32(0, n), n, True)
    call = lambda cu: fresh(lambda: fa.forward_varlen_prefill_fp16(q, k, v, cu, n, True), one)
    assert not wrong(call(i32(0, *[n, 0] * times, n)), one)
    # rows that only the first sequence has come last, among the lightest items
    first = fa.forward_varlen_prefill_fp16(*(t[600:].contiguous() for t in (q, k, v)), i32(0, 100), n, True)
    rest = fa.forward_varlen_prefill_fp16(*(t[:600].contiguous() for t in (q, k, v)), i32(0, 600), n, True)
    got = call(i32(600, 700, *[0, 600] * times))
    assert not wrong(got[600:], first) and not wrong(got[:600], rest)
