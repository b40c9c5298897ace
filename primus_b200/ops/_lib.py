"""Python binding of ``libprimus_b200.so`` (the sm_100a kernels under ``primus_b200/csrc``): the launchers are called through a
compiled module (``csrc/python/launch.c``), or through ctypes where that is not built or does not load.

The library exports ``extern "C"`` launchers that take raw device pointers and a CUDA stream.
``call(name, *args)`` converts torch tensors to pointers, appends nothing implicitly, and raises
on a non-zero return code.  On a machine with a GPU the library is mandatory: ops never fall back
to PyTorch for CUDA tensors (``require()`` raises if the library is missing).
"""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import os
import sys
import sysconfig
import threading
import warnings
from pathlib import Path

import torch

_LIB = None
_LOCK = threading.Lock()
LIB_PATH = Path(__file__).resolve().parent.parent / "lib" / "libprimus_b200.so"


class NativeLibraryError(RuntimeError):
    pass


def lib_path() -> Path:
    return Path(os.environ.get("PRIMUS_B200_LIB", LIB_PATH))


def available() -> bool:
    return lib_path().exists()


def load():
    """Load (once) and return the ctypes handle."""
    global _LIB
    if _LIB is None:
        with _LOCK:
            if _LIB is None:
                p = lib_path()
                if not p.exists():
                    raise NativeLibraryError(
                        f"{p} not found: build it with `python -m primus_b200.build` "
                        "(CUDA tensors are never routed to a PyTorch fallback)"
                    )
                _LIB = ctypes.CDLL(str(p), mode=ctypes.RTLD_GLOBAL)
    return _LIB


def require():
    return load()


_PTR = ctypes.c_void_p


def stream_ptr() -> ctypes.c_void_p:
    return _PTR(torch.cuda.current_stream().cuda_stream)


def _ctype(a):
    """C type an argument travels as: floats single precision, integers 64-bit (a launcher's 32-bit parameter reads the low
    half of the register), single ctypes values their own type.  All else is a pointer: tensors, None, and ctypes arrays,
    which as their own class would admit no other length."""
    if isinstance(a, float):
        return ctypes.c_float
    if isinstance(a, int):
        return ctypes.c_long
    if isinstance(a, ctypes._SimpleCData):
        return type(a)
    return _PTR


def _load_launch():
    """The compiled binding beside the library, or None: calls then go through ctypes."""
    path = LIB_PATH.parent / ("_launch" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))
    if not path.exists():
        return None
    try:
        loader = importlib.machinery.ExtensionFileLoader("_launch", str(path))
        module = importlib.util.module_from_spec(importlib.util.spec_from_loader("_launch", loader))
        loader.exec_module(module)
        module.init(torch.Tensor)
    except ImportError as e:
        warnings.warn(f"{path} does not load ({e}): launchers are called through ctypes")
        return None
    return module


_LAUNCH = _load_launch()

# Launchers bound so far: name -> (function of (arguments, stream), kernels per call).  The kinds of a launcher's arguments are
# those of its first call; an integer in a float's place is converted.  A later call may bring an argument of another kind
# (None after an integer, a ctypes integer after a plain one): it is refused before anything is called, and the launcher is
# bound anew.
_BOUND: dict = {}


def _ctypes_launcher(fn, argtypes, stream: bool):
    """What the compiled binding does, through ctypes: for ctypes values, and where the binding is not built."""
    fn.restype = ctypes.c_int
    fn.argtypes = argtypes + ([_PTR] if stream else [])

    def launch(args, stream_ptr):
        plain = [a.data_ptr() if isinstance(a, torch.Tensor) else a for a in args]
        if stream:
            plain.append(stream_ptr)
        try:
            return fn(*plain)
        except ctypes.ArgumentError:
            return None

    return launch


_tracing = torch._C._is_tracing


def _bind(name: str, args, stream: bool):
    if _tracing() and any(isinstance(a, torch.Tensor) and not a.dim() and not a.is_cuda for a in args):
        # (what a recorded shape consists of: its address would travel in the number's place)
        raise NativeLibraryError(f"pb_{name}: sizes are tensors while torch.jit.trace records")
    fn = load()["pb_" + name]       # an object of its own: argument types set here are not seen by other users
    launch = None
    if _LAUNCH is not None and all(a is None or isinstance(a, (torch.Tensor, int, float, bytes)) for a in args):
        kinds = "".join("f" if isinstance(a, float) else "l" if isinstance(a, int) else "p" for a in args)
        launch = _LAUNCH.bind(ctypes.cast(fn, _PTR).value, kinds.encode(), stream)
    if launch is None:
        launch = _ctypes_launcher(fn, [_ctype(a) for a in args], stream)
    _BOUND[name, stream] = bound = (launch, _KERNELS_PER_CALL.get(name, 1))
    return bound


# Number of device kernels each launcher enqueues (default 1); used for the launch counter below.
_KERNELS_PER_CALL = {"rmsnorm_bwd": 2, "rmsnorm_bwd_two": 2, "rmsnorm_bwd_y": 2, "sumsq": 2, "grad_norm": 2, "flash_attn_bwd": 3, "flash_attn_bwd_cap": 3, "quant_fp8_tensorwise": 2,
                     "quant_fp8_delayed": 2, "gemm_bf16_splitk": 2, "qk_norm_rope_bwd": 3}
LAUNCH_COUNT = 0


def _bound_anew(name: str, args, stream: bool, stream_ptr: int) -> int:
    rc = _bind(name, args, stream)[0](args, stream_ptr)
    if rc is None:
        raise ctypes.ArgumentError(f"pb_{name}: an argument cannot be passed: {args}")
    return rc


def call(name: str, *args) -> None:
    """Invoke ``pb_<name>`` with converted arguments; the current CUDA stream is appended."""
    global LAUNCH_COUNT
    launch, kernels = _BOUND.get((name, True)) or _bind(name, args, True)
    LAUNCH_COUNT += kernels
    stream = torch._C._cuda_getCurrentRawStream(torch.cuda.current_device())
    rc = launch(args, stream)
    if rc is None:
        rc = _bound_anew(name, args, True, stream)
    if rc != 0:
        raise NativeLibraryError(f"pb_{name} failed with code {rc}")


def call_ret(name: str, *args) -> int:
    """Invoke a host-only helper that returns a value (no stream appended)."""
    launch, _ = _BOUND.get((name, False)) or _bind(name, args, False)
    rc = launch(args, 0)
    return _bound_anew(name, args, False, 0) if rc is None else rc


def _load_nodes():
    """The C++ autograd nodes beside the library, or None: the layers then run as Python functions.  The file's name says which
    torch and which launchers a module was compiled for; none of another name is opened."""
    from ..build import nodes_name

    if not available() or not torch.cuda.is_available():
        return None
    try:
        answer = load().pb_abi
        answer.restype = ctypes.c_char_p
        path = LIB_PATH.parent / nodes_name(torch.__version__, answer().decode())
    except AttributeError:                      # a library without an answer: an older one
        path = LIB_PATH.parent / "none"
    if not path.exists():
        others = sorted(p.name for p in LIB_PATH.parent.glob("_nodes*"))
        if others:
            warnings.warn(f"{', '.join(others)}: not for torch {torch.__version__} and the launchers of {lib_path()} "
                          "(python -m primus_b200.build); layers run as Python functions")
        return None
    from . import autotune, gemm

    try:
        loader = importlib.machinery.ExtensionFileLoader("_nodes", str(path))
        module = importlib.util.module_from_spec(importlib.util.spec_from_loader("_nodes", loader))
        loader.exec_module(module)
        module.init(str(lib_path()), sys.modules[__name__], gemm, autotune)
    except (ImportError, RuntimeError) as e:
        warnings.warn(f"{path} does not load ({e}): layers run as Python functions")
        return None
    return module


_NODES: list = []       # [the module, or None]


_PLAIN = (torch.Tensor, torch.nn.Parameter)
_functorch = torch._C._are_functorch_transforms_active


def nodes(*tensors):
    """The C++ autograd nodes where they take these tensors (bf16 on the GPU, no subclass, no function transform or trace at work; None
    among them counts as taken), else None."""
    if not _NODES:
        _NODES.append(_load_nodes())
    n = _NODES[0]
    if n is None or _functorch() or _tracing():
        return None
    for t in tensors:
        if t is not None and (type(t) not in _PLAIN or t.dtype is not torch.bfloat16 or not t.is_cuda):
            return None
    return n


def launch_count() -> int:
    """Kernels launched so far, from Python and by the C++ nodes."""
    return LAUNCH_COUNT + (_NODES[0].launches() if _NODES and _NODES[0] is not None else 0)


class I32(int):
    """Marks a Python int that must be passed as a 32-bit int."""


def i32(x: int):
    return ctypes.c_int(int(x))


# ---------------------------------------------------------------------------------------------
# Device status word: kernels with bounded waits report a timeout here instead of hanging.
_STATUS: dict[int, torch.Tensor] = {}

STATUS_MESSAGES = {
    0: "ok",
    1: "TMA producer timed out waiting for a free shared-memory stage",
    2: "MMA issuer timed out waiting for operands or an accumulator slot",
    3: "epilogue timed out waiting for an accumulator",
    4: "timed out waiting for a peer flag in global memory",
    5: "bad argument detected on the device",
    6: "routed rows exceed the capacity of the expert-parallel buffers (raise moe_fused_capacity_factor)",
}


def status_word(device: torch.device | int | None = None) -> torch.Tensor:
    dev = torch.cuda.current_device() if device is None else torch.device(device).index or 0
    t = _STATUS.get(dev)
    if t is None:
        t = torch.zeros(1, dtype=torch.int32, device=f"cuda:{dev}")
        _STATUS[dev] = t
    return t


def check_status(device=None) -> None:
    """Synchronising check of the device status word; raises if a kernel recorded an error."""
    t = status_word(device)
    code = int(t.item())
    if code != 0:
        t.zero_()
        raise NativeLibraryError(f"device kernel reported status {code}: {STATUS_MESSAGES.get(code, '?')}")
