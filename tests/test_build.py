"""What the build needs, and what it may not take for granted (no GPU)."""
import os
import sysconfig
import types

import pytest
import torch

from flexllm_b200 import build, ops


@pytest.mark.parametrize("how", ["fails", "missing"])
def test_library_is_built_without_the_extension(monkeypatch, tmp_path, how):
    """No compiler or no headers for the Python extension: a warning, the library, and no file in the extension's place."""
    build.build_library()
    out = str(tmp_path / "ext.so")
    monkeypatch.setattr(build, "front_end_path", lambda: out)

    def run(cmd, **kw):
        if how == "missing":
            raise FileNotFoundError(cmd[0])
        open(cmd[cmd.index("-o") + 1], "w").write("half")
        return types.SimpleNamespace(returncode=1, stdout="", stderr="Python.h: No such file or directory")
    monkeypatch.setattr(build.subprocess, "run", run)
    with pytest.warns(UserWarning, match="front end"):
        assert build.build() == build.LIB
    assert not os.listdir(tmp_path)


def test_extension_of_another_torch_or_python_is_not_loaded(monkeypatch):
    assert torch.__version__ in build.front_end_path() and build.front_end_path().endswith(sysconfig.get_config_var("EXT_SUFFIX"))
    build.build()
    monkeypatch.setattr(ops, "_front", None)
    assert ops._bind_front_end()
    monkeypatch.setattr(ops, "_front", None)
    monkeypatch.setattr(torch, "__version__", "0.1")
    assert not ops._bind_front_end()
