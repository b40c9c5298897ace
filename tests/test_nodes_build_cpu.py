"""The C++ autograd nodes are loaded for the torch and the launchers that they were compiled for, and for no others."""
import ctypes
import shutil
import subprocess
import sysconfig

import pytest
import torch

from primus_b200 import build
from primus_b200.ops import _lib

SUFFIX = sysconfig.get_config_var("EXT_SUFFIX") or ".so"


def _nodes(monkeypatch):
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    return _lib._load_nodes()


@pytest.fixture
def built(monkeypatch):
    if not _lib.available() or not list(build.LIB_DIR.glob("_nodes-*" + SUFFIX)):
        pytest.skip("the library or the autograd nodes are not built")
    assert _nodes(monkeypatch) is not None


def test_name_is_that_of_the_build(built):
    answer = _lib.load().pb_abi
    answer.restype = ctypes.c_char_p
    assert answer().decode() == build.launcher_abi() and build._torch_version() == torch.__version__


def test_another_torch(built, monkeypatch):
    monkeypatch.setattr(torch, "__version__", "2.99.0")
    with pytest.warns(UserWarning, match="Python functions"):
        assert _nodes(monkeypatch) is None


@pytest.mark.parametrize("source", ['extern "C" const char* pb_abi() { return "0123"; }', 'extern "C" int pb_other() { return 0; }'])
def test_other_launchers(built, monkeypatch, tmp_path, source):
    (tmp_path / "l.cpp").write_text(source)
    subprocess.run(["g++", "-shared", "-fPIC", str(tmp_path / "l.cpp"), "-o", str(tmp_path / "l.so")], check=True)
    monkeypatch.setattr(_lib, "_LIB", ctypes.CDLL(str(tmp_path / "l.so")))
    with pytest.warns(UserWarning, match="Python functions"):
        assert _nodes(monkeypatch) is None


def test_declarations_make_the_name(monkeypatch, tmp_path):
    for f in build._sources():
        shutil.copy(f, tmp_path)
    monkeypatch.setattr(build, "CSRC", tmp_path)
    src = tmp_path / "router.cu"
    before, text = build.launcher_abi(), src.read_text()
    src.write_text(text + "\n// a comment\n")
    assert build.launcher_abi() == before
    src.write_text(text.replace("int pb_moe_route(const void* logits, int in_bf16,", "int pb_moe_route(int in_bf16, const void* logits,"))
    assert build.launcher_abi() != before


@pytest.mark.parametrize("version", ["2.99.0", ""])
def test_build_leaves_no_other_module_behind(monkeypatch, tmp_path, capsys, version):
    stale = [tmp_path / ("_nodes" + SUFFIX), tmp_path / build.nodes_name("1.0", "0123")]
    for f in stale:
        f.write_bytes(b"")
    monkeypatch.setattr(build, "LIB_DIR", tmp_path)
    monkeypatch.setattr(build, "_torch_version", lambda: version)
    monkeypatch.setenv("PATH", str(tmp_path))                      # no compiler
    monkeypatch.setenv("NVCC", str(tmp_path / "_nodes"))
    (tmp_path / "_nodes").write_bytes(b"")
    build._build_nodes(force=False)
    assert not any(f.exists() for f in stale) and "Python functions" in capsys.readouterr().err
    assert not (tmp_path / build.nodes_name(version, build.launcher_abi())).exists()
