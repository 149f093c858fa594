"""GPU: the native host side of the calls (csrc/host/call.cpp) against the Python one: the same results bit for bit on the plain case, and every other
call handed back to Python, which then does or refuses what it always did."""
import pytest
import torch

from flash_attn_v100_b200 import ops

pytestmark = pytest.mark.gpu
H, BF = torch.float16, torch.bfloat16


def rnd(*shape, dtype=H):
    return torch.randn(*shape, device="cuda").to(dtype)


def calls(dtype=H):
    """name -> (operator, its arguments)."""
    q, k, v = rnd(3, 8, 1, 64, dtype=dtype), rnd(3, 2, 48, 64, dtype=dtype), rnd(3, 2, 48, 64, dtype=dtype)
    i32 = lambda *x: torch.tensor(x, dtype=torch.int32, device="cuda")
    pages = [rnd(9, 2, 16, 64, dtype=dtype) for _ in range(2)]
    table, lens = torch.randperm(9, device="cuda").to(torch.int32).view(3, 3), i32(5, 0, 48)
    packed = [rnd(70, h, 64, dtype=dtype) for h in (8, 2, 2)]
    dense = [rnd(2, h, 33, 64, dtype=dtype) for h in (8, 2, 2)]
    cu = i32(3, 20, 20, 61)
    if dtype == BF:
        return dict(decode=(ops.forward_decode_gqa_bf16, (q, k, v, True, 40)), paged=(ops.forward_paged_decode_gqa_bf16, (q, *pages, table, lens, 3)),
                    dense=(ops.forward_prefill_gqa_bf16, (*dense, True)), varlen=(ops.forward_varlen_prefill_bf16, (*packed, cu, 41, True)))
    k8, v8 = (torch.randint(-127, 128, (3, 2, 48, 64), device="cuda", dtype=torch.int8) for _ in range(2))
    s = [(torch.rand(3, 2, 48, device="cuda") * 0.02 + 0.01).to(t) for t in (H, H, torch.float32)]
    return dict(decode=(ops.forward_decode_gqa_fp16, (q, k, v, True, 40)), paged=(ops.forward_paged_decode_gqa_fp16, (q, *pages, table, lens, 3)),
                contig=(ops.forward_continuous_batching_fp16, (q, k, v, i32(4, 0, 47), True)),
                window=(ops.forward_decode_sliding_window_gqa, (q, k, v, True, 40, 17, 3)), int8_kv=(ops.forward_decode_int8_kv_cache_gqa, (q, k8, v8, s[0], s[1], 40)),
                int8_qk=(ops.forward_decode_int8_gqa, (q, k, v, rnd(3, 8).abs().float() * 0.02 + 0.01, s[2], 40)),
                dense=(ops.forward_prefill_gqa_fp16, (*dense, False)), varlen=(ops.forward_varlen_prefill_fp16, (*packed, cu, 41, False)))


CASES = [(H, n) for n in ("decode", "paged", "contig", "window", "int8_kv", "int8_qk", "dense", "varlen")] + \
    [(BF, n) for n in ("decode", "paged", "dense", "varlen")]


@pytest.fixture
def log(monkeypatch):
    """Which calls the native side took."""
    taken, native = [], ops._native

    def spy(name, *args):
        out = native(name, *args)
        taken.append((name, out is not None))
        return out
    monkeypatch.setattr(ops, "_native", spy)
    return taken


def python_only(monkeypatch, f, args):
    with monkeypatch.context() as m:
        m.setattr(ops, "_native", lambda *a: None)
        return f(*args)


@pytest.mark.parametrize("dtype,name", CASES)
def test_same_bits_as_the_python_side(log, monkeypatch, dtype, name):
    torch.manual_seed(1)
    f, args = calls(dtype)[name]
    ref = python_only(monkeypatch, f, args)
    out = f(*args)
    assert log[-1] == (name, True)
    assert out.shape == ref.shape and out.dtype == ref.dtype and torch.equal(out, ref)


class Sub(torch.Tensor):
    pass


@pytest.mark.parametrize("dtype,name", CASES)
def test_other_calls_go_back_to_python(log, monkeypatch, dtype, name):
    """A tensor subclass, a function mode and a number that is not a plain one are served as before; a layout, a type or a device that does not fit is refused as
    before, with the same message."""
    torch.manual_seed(2)
    f, args = calls(dtype)[name]
    ref = python_only(monkeypatch, f, args)
    assert torch.equal(f(args[0].as_subclass(Sub), *args[1:]).as_subclass(torch.Tensor), ref) and not log[-1][1]
    with torch.device("cuda"):                                     # a function mode
        assert torch.equal(f(*args), ref) and not log[-1][1]
    if isinstance(args[-1], int) and not isinstance(args[-1], bool):
        assert torch.equal(f(*args[:-1], torch.tensor(args[-1])), ref) and not log[-1][1]
    wrong = [args[1].transpose(0, 1), args[1].float(), args[1].cpu(), args[1][..., :56].contiguous(), args[1][None]]
    for t in wrong:
        messages = []
        for call in (lambda: f(args[0], t, *args[2:]), lambda: python_only(monkeypatch, f, (args[0], t, *args[2:]))):
            with pytest.raises(RuntimeError) as e:
                call()
            messages.append(str(e.value))
        assert messages[0] == messages[1]


def test_vmap_is_refused_as_before():
    f, args = calls()["decode"]
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda q: f(q, *args[1:]))(args[0][None])


def test_first_call_of_a_stream_and_growth(log):
    """No scratch for a stream yet: Python makes it, and the next call is native; a larger batch outgrows it and gets a new one."""
    f, args = calls()["decode"]
    ref = f(*args)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        outs = [f(*args), f(*args)]
        big = [rnd(4096, 2, 1, 64), rnd(4096, 2, 16, 64), rnd(4096, 2, 16, 64)]
        outs.append(f(*big, True, 15))
        outs.append(f(*args))
    s.synchronize()
    native = [ok for name, ok in log]
    assert not native[1] and native[2] and native[-1]
    assert all(torch.equal(o, ref) for o in (outs[0], outs[1], outs[3]))


def test_captured_and_from_two_threads(log):
    import threading
    f, args = calls()["paged"]
    ref = f(*args)
    g = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        f(*args)
    torch.cuda.current_stream().wait_stream(s)
    with torch.cuda.graph(g, stream=s):
        out = f(*args)
    assert log[-1] == ("paged", True)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, ref)
    bad = []

    def work():
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(50):
                if not torch.equal(f(*args), ref):
                    bad.append(1)
    threads = [threading.Thread(target=work) for _ in range(2)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not bad
