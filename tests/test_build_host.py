"""When the native launcher is built again (no compiler runs here)."""

import importlib.util
import os
import subprocess
import sys
import types

import pytest
import torch

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flash-sparse-attention_b200")


def test_rebuilt_when_what_it_was_built_with_changes(monkeypatch, tmp_path):
    spec = importlib.util.spec_from_file_location("fsa_build", os.path.join(PKG, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    lib = tmp_path / "_host.so"
    monkeypatch.setattr(build, "HOST_LIB", str(lib))
    monkeypatch.setattr(build, "OBJ", str(tmp_path / "objects"))
    runs = []

    def run(cmd, **kw):
        runs.append(cmd)
        with open(cmd[cmd.index("-o") + 1], "w") as f:
            f.write(str(len(runs)))
        return types.SimpleNamespace(returncode=fail, stdout="", stderr="no")

    fail = 0
    monkeypatch.setattr(subprocess, "run", run)
    build.build_host()
    build.build_host()
    assert len(runs) == 1 and lib.read_text() == "1"
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    build.build_host()
    assert len(runs) == 2 and lib.read_text() == "2"
    monkeypatch.setattr(sys, "version", "another interpreter")
    fail = 1
    with pytest.raises(RuntimeError, match="fsa_host"):
        build.build_host()
    assert lib.read_text() == "2"  # a failed build leaves the module that is there
    fail = 0
    build.build_host()
    build.build_host()
    assert len(runs) == 4 and lib.read_text() == "4"
