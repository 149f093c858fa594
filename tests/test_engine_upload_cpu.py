"""The engine's host vectors travel in one buffer: each arrives whole, at an aligned place."""
import pytest
import torch

from flash_attn_v100_b200.engine.runner import _upload


@pytest.mark.parametrize("sizes", [(1, 1), (3, 0, 5), (17, 16, 1, 33), (0,)])
def test_parts_arrive_whole_and_aligned(sizes):
    parts = [torch.arange(n, dtype=torch.int64 if i % 2 == 0 else torch.int32) * 3 - i for i, n in enumerate(sizes)]
    got = _upload(parts, torch.device("cpu"))
    assert [t.dtype for t in got] == [t.dtype for t in parts]
    for g, p in zip(got, parts):
        assert torch.equal(g, p)
        assert g.numel() == 0 or (g.data_ptr() - got[0].data_ptr()) % 64 == 0
