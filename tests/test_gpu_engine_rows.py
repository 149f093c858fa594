"""GPU: a prompt pass whose last layer goes on with the wanted rows only, against the oracle's logits at those places: the last ones, any others, some of them
twice and out of order, all of them, none of one prompt; and the tokens decoded behind it read the cache of all tokens."""
import pytest
import torch

from tests.test_gpu_engine import TOL, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("places", [([20], [6]), ([0, 20, 7], [6]), ([3, 3, 1], [5, 0]), (list(range(21)), list(range(7))), ([], [6])])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_wanted_rows(places, dtype):
    from oracle import model_oracle as mo
    cfg, model, Runner = _setup()
    model.attn_dtype = dtype
    g = torch.Generator().manual_seed(4)
    prompts = [torch.randint(0, cfg.vocab_size, (n,), generator=g) for n in (21, 7)]
    runner = Runner(model, max_batch=2, max_seq_len=64)
    for r in "ab":
        runner.start(r)
    out = runner.step([(r, p.tolist(), w) for r, p, w in zip("ab", prompts, places)])
    nxt = runner.step([(r, [int(p[0])], [0]) for r, p in zip("ab", prompts)])
    runner.check_errors()
    for p, w, logits, after in zip(prompts, places, out, nxt):
        ref = mo.forward_logits(cfg, 5, torch.cat([p, p[:1]])[None])[0]
        assert logits.shape == (len(w), cfg.vocab_size)
        if w:
            assert (logits.cpu() - ref[w]).abs().max() < TOL
        assert (after.cpu() - ref[-1:]).abs().max() < TOL
