"""Builds the native library (``primus_b200/lib/libprimus_b200.so``) from ``primus_b200/csrc``.

All device code targets sm_100a only (``-gencode arch=compute_100a,code=sm_100a``); nvcc
cross-compiles it on hosts without a GPU.  The library exposes plain ``extern "C"`` launchers
(raw pointers + a CUDA stream) that :mod:`primus_b200.ops._lib` calls through a small CPython module
(``csrc/python/launch.c``, compiled with gcc; ctypes without it), so a rebuild of the kernels takes seconds and no torch headers.
Those are needed by one module alone, the C++ autograd nodes of the common layers (``csrc/python/nodes.cpp``), which is compiled
beside the kernels.

Run ``python -m primus_b200.build`` (add ``--force`` to rebuild everything, ``--verbose`` to see
ptxas resource usage).
"""
from __future__ import annotations

import argparse
import concurrent.futures
import hashlib
import importlib.util
import os
import platform
import re
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
LIB_DIR = PKG_DIR / "lib"
OBJ_DIR = LIB_DIR / "obj"
LIB_PATH = LIB_DIR / "libprimus_b200.so"
# the launchers' Python binding; its name says which interpreter it is for
LAUNCH_SRC = CSRC / "python" / "launch.c"
LAUNCH_PATH = LIB_DIR / ("_launch" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))
# autograd nodes of the common layers (torch headers: half a minute)
NODES_SRC = CSRC / "python" / "nodes.cpp"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "--expt-relaxed-constexpr",
    "-Xcompiler", "-fPIC",
    "-Xcompiler", "-fvisibility=default",
]


def nodes_name(torch_version: str, abi: str) -> str:
    """File name of the autograd nodes: which torch they were compiled for, which launchers they call and which interpreter they
    are for, so that nothing else is ever loaded."""
    return f"_nodes-torch{torch_version}-{abi}{sysconfig.get_config_var('EXT_SUFFIX') or '.so'}"


def launcher_abi() -> str:
    """What the launchers' declarations hash to.  The library answers with it to ``pb_abi``."""
    declarations = []
    for src in _sources():
        declarations += re.findall(r"^(?:extern\s+\"C\"\s+)?(\w[\w\s*]*?\bpb_\w+\s*\([^)]*\))\s*\{", src.read_text(), re.M)
    return hashlib.sha256("\n".join(sorted(" ".join(d.split()) for d in declarations)).encode()).hexdigest()[:12]


def _torch_version() -> str:
    """Without importing it; empty where there is none."""
    spec = importlib.util.find_spec("torch")
    if spec is None or not spec.submodule_search_locations:
        return ""
    text = (Path(spec.submodule_search_locations[0]) / "version.py").read_text()
    return re.search(r"""^__version__\s*=\s*['"]([^'"]+)""", text, re.M).group(1)


def find_nvcc() -> str:
    cand = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(cand).exists():
        raise RuntimeError("nvcc not found; set NVCC or install the CUDA toolkit")
    return cand


def _sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cpp"))


def _needs_build(src: Path, obj: Path, headers: list[Path]) -> bool:
    if not obj.exists():
        return True
    t = obj.stat().st_mtime
    return src.stat().st_mtime > t or any(h.stat().st_mtime > t for h in headers)


def _compile_one(nvcc: str, src: Path, obj: Path, verbose: bool) -> tuple[Path, int, str]:
    cmd = [nvcc, *NVCC_FLAGS, "-I", str(CSRC), "-c", str(src), "-o", str(obj)]
    if src.suffix == ".cpp":
        cmd = [nvcc, "-O2", "-std=c++17", "-Xcompiler", "-fPIC", "-I", str(CSRC), "-c", str(src), "-o", str(obj)]
    elif verbose:
        cmd[1:1] = ["-Xptxas", "-v"]
    p = subprocess.run(cmd, capture_output=True, text=True)
    return src, p.returncode, p.stdout + p.stderr


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile out-of-date sources and link the shared library. Returns the library path."""
    with concurrent.futures.ThreadPoolExecutor(1) as beside:
        nodes = beside.submit(_build_nodes, force)
        _build_library(force, verbose)
        _build_launch(force)
        nodes.result()
    return LIB_PATH


def _build_library(force: bool, verbose: bool) -> None:
    nvcc = find_nvcc()
    OBJ_DIR.mkdir(parents=True, exist_ok=True)
    abi = OBJ_DIR / "abi.cpp"
    text = f'extern "C" const char* pb_abi() {{ return "{launcher_abi()}"; }}\n'
    if not abi.exists() or abi.read_text() != text:
        abi.write_text(text)
    headers = sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.h"))
    jobs = []
    objs = []
    for src in [*_sources(), abi]:
        obj = OBJ_DIR / (src.name + ".o")
        objs.append(obj)
        if force or _needs_build(src, obj, headers):
            jobs.append((src, obj))
    if jobs:
        with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            results = list(ex.map(lambda so: _compile_one(nvcc, so[0], so[1], verbose), jobs))
        failed = [(s, out) for s, rc, out in results if rc != 0]
        if verbose:
            for s, rc, out in results:
                print(f"--- {s.name}\n{out}")
        if failed:
            msg = "\n".join(f"{s}:\n{out}" for s, out in failed)
            raise RuntimeError(f"nvcc failed:\n{msg}")
    if jobs or not LIB_PATH.exists():
        cmd = [nvcc, "-shared", "-o", str(LIB_PATH), *map(str, objs), "-lcudart", "-ldl"]
        p = subprocess.run(cmd, capture_output=True, text=True)
        if p.returncode != 0:
            raise RuntimeError(f"link failed:\n{p.stdout}{p.stderr}")


def _build_launch(force: bool) -> None:
    """The launchers' binding.  Where it cannot be built (another architecture, no headers of Python, no gcc), calls go through
    ctypes; a binding of an older source does not stay behind."""
    include = Path(sysconfig.get_paths()["include"])
    if not force and not _needs_build(LAUNCH_SRC, LAUNCH_PATH, []):
        return
    if platform.machine() != "x86_64" or not (include / "Python.h").exists():
        why = "Python headers for x86-64 not found"
    else:
        cmd = ["gcc", "-O2", "-shared", "-fPIC", "-I", str(include), str(LAUNCH_SRC), "-o", str(LAUNCH_PATH)]
        try:
            p = subprocess.run(cmd, capture_output=True, text=True)
            if p.returncode == 0:
                return
            why = f"the compiled binding could not be built:\n{p.stdout}{p.stderr}"
        except OSError as e:
            why = f"the compiled binding could not be built ({e})"
    LAUNCH_PATH.unlink(missing_ok=True)
    print(f"{why}\nlaunchers are called through ctypes", file=sys.stderr)


def _build_nodes(force: bool) -> None:
    """The C++ autograd nodes.  Where they cannot be built, the layers run as Python functions; a module of an older source, of
    another torch or for other launchers does not stay behind."""
    version = _torch_version()
    path = LIB_DIR / nodes_name(version, launcher_abi())
    for other in LIB_DIR.glob("_nodes*" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so")):
        if other != path:
            other.unlink(missing_ok=True)
    if not force and not _needs_build(NODES_SRC, path, []):
        return
    path.unlink(missing_ok=True)
    if platform.machine() != "x86_64" or not version:
        why = "x86-64 and torch are needed"
    else:
        import torch

        LIB_DIR.mkdir(parents=True, exist_ok=True)
        root, cuda = Path(torch.__file__).parent, Path(find_nvcc()).parent.parent
        includes = [root / "include", root / "include/torch/csrc/api/include", cuda / "include", sysconfig.get_paths()["include"]]
        cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_nodes",
               f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", *[f"-I{i}" for i in includes], str(NODES_SRC),
               "-o", str(path), f"-L{root / 'lib'}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"]
        try:
            p = subprocess.run(cmd, capture_output=True, text=True)
            if p.returncode == 0:
                return
            why = f"{p.stdout}{p.stderr}"
        except OSError as e:
            why = str(e)
    path.unlink(missing_ok=True)
    print(f"the autograd nodes could not be built:\n{why}\nlayers run as Python functions", file=sys.stderr)


def main() -> None:
    ap = argparse.ArgumentParser(description=__doc__)
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    path = build(force=a.force, verbose=a.verbose)
    print(path)


if __name__ == "__main__":
    sys.exit(main())
