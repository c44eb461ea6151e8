"""The build script: when the host extension is built again, and without torch."""
import importlib.util
import os
import types

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture
def build(tmp_path, monkeypatch):
    spec = importlib.util.spec_from_file_location("ctb_build_test", os.path.join(ROOT, "cutile.jl_b200", "csrc", "build.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    monkeypatch.setattr(mod, "HOST", str(tmp_path / "_host.so"))
    monkeypatch.setattr(mod, "OBJ_DIR", str(tmp_path))
    mod.runs = []

    def run(cmd, **kw):
        mod.runs.append(cmd)
        open(mod.HOST, "w").close()
        return types.SimpleNamespace(returncode=0, stdout="", stderr="")
    monkeypatch.setattr(mod.subprocess, "run", run)
    return mod


def test_host_extension_follows_torch(build, monkeypatch):
    import torch
    build.build_host()
    build.build_host()
    assert len(build.runs) == 1 and f'-DCTB_TORCH_VERSION="{torch.__version__}"' in build.runs[0]
    env = dict(build.built_for(), torch="0.0.1")
    monkeypatch.setattr(build, "built_for", lambda: env)
    build.build_host()
    assert len(build.runs) == 2 and '-DCTB_TORCH_VERSION="0.0.1"' in build.runs[1]
    env["python"] = "cpython-399"
    build.build_host()
    build.build_host()
    assert len(build.runs) == 3


def test_without_torch_only_the_c_library_is_built(build, monkeypatch, capsys):
    monkeypatch.setattr(build.importlib.util, "find_spec", lambda name: None)
    build.build_host(force=True)
    assert build.runs == [] and "torch is not installed" in capsys.readouterr().err


def test_the_extension_names_its_torch():
    import torch

    from cutile_b200 import _host
    assert _host.TORCH_VERSION == torch.__version__
