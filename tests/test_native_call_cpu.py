"""The native host side of the calls is built, fits the installed torch, and hands back what is not for it."""
import shutil

import pytest
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


def test_module_for_another_torch_is_built_again_and_not_loaded(monkeypatch, tmp_path):
    """As the sources are no younger, only what it was built for tells: here the installed torch is another one."""
    from flash_attn_v100_b200 import build
    path = build.build_call()
    assert build.call_fits(path)
    built = []
    monkeypatch.setattr(torch, "__version__", "9.9.9+cu000")
    assert not build.call_fits(path)
    with pytest.warns(RuntimeWarning, match="built for another torch"):
        assert _lib.call_module(ops._workspaces) is None
    monkeypatch.setattr(build, "_run", lambda cmd: built.append(cmd) or open(cmd[cmd.index("-o") + 1], "w").close())
    monkeypatch.setattr(build, "CALL_PATH", str(tmp_path / "_call.so"))
    shutil.copy2(path, tmp_path / "_call.so")
    build.build_call()
    assert len(built) == 1 and any("9.9.9+cu000" in a for a in built[0])


def test_build_without_a_host_compiler_keeps_the_libraries(monkeypatch):
    from flash_attn_v100_b200 import build

    def no_compiler(force):
        raise FileNotFoundError("g++")
    monkeypatch.setattr(build, "build", lambda force, verbose, library: library)
    monkeypatch.setattr(build, "build_call", no_compiler)
    with pytest.warns(RuntimeWarning, match="g\\+\\+"):
        assert build.build_all() == list(build.LIBRARIES)
