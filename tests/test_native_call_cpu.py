"""The native host side of the calls is built, fits the installed torch, and hands back what is not for it."""
import torch

from flash_attn_v100_b200 import _lib, ops
from flash_attn_v100_b200.build import build_call


def test_built_and_bound():
    build_call()
    mod = _lib.call_module(ops._workspaces)
    assert mod is not None and mod.torch_version == torch.__version__.split("+")[0]


def test_cpu_tensors_are_handed_back():
    mod = _lib.call_module(ops._workspaces)
    q, k = torch.zeros(1, 2, 1, 64, dtype=torch.float16), torch.zeros(1, 2, 16, 64, dtype=torch.float16)
    assert mod.decode(q, k, k, True, 3, False) is None
    assert mod.decode(q, k) is None
    assert mod.dense(None, None, None, True, False) is None
