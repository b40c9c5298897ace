"""Host-side parts of the native library and of its binding, on a machine without a GPU."""
import contextlib
import ctypes
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from primus_b200 import build
from primus_b200.ops import _lib, attention, fused, layers

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "primus_b200" / "csrc"


def _compile(tmp_path, name, source, *flags):
    src, out = tmp_path / f"{name}.cpp", tmp_path / name
    src.write_text(source)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), *flags, str(src), "-o", str(out)], check=True)
    return out


DIVISION = r"""
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "div_invariant.h"

static float bits(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
static uint32_t bits(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }

// differences (in bits; any NaN equals any other) from the division over `count` numerators from `first`, `step` apart
static long differ(float b, uint32_t first, uint32_t step, uint32_t count) {
  const float r = (float)(1.0 / b);
  long bad = 0;
  for (uint32_t i = 0; i < count; ++i) {
    const float a = bits(first + i * step), got = pb::div_invariant(a, b, r), want = a / b;
    bad += (bits(got) != bits(want)) & !((got != got) & (want != want));
  }
  return bad;
}

int main(int argc, char** argv) {
  for (int i = 1; i < argc; ++i) {
    const float b = (float)atof(argv[i]);
    const long mantissas = differ(b, bits(1.f), 1, 1u << 23);                  // every mantissa of one binade
    const long range = differ(b, 0, 1021, 0xffffffffu / 1021);                 // signs, subnormals, infinities, NaN
    const long small = differ(b, 0, 1, 1u << 20) + differ(b, 0x80000000u, 1, 1u << 20) + differ(b, bits(0x1p-101f), 3, 1u << 22);
    const long large = differ(b, bits(0x1p125f), 5, (bits(INFINITY) - bits(0x1p125f)) / 5);
    if (mantissas || range || small || large)
      printf("b = %.9g: %ld mantissas, %ld over the range, %ld small, %ld large\n", b, mantissas, range, small, large);
  }
}
"""


def test_division_by_an_invariant_is_the_division(tmp_path):
    """Bias corrections 1 - beta^step as the optimizer kernels get them, and divisors around which an estimate rounds badly."""
    exe = _compile(tmp_path, "division", DIVISION, "-O3", "-march=native", "-ffp-contract=off")
    corrections = [1.0 - beta ** step for beta in (0.9, 0.95, 0.99, 0.999) for step in (1, 2, 3, 10, 100, 1000)]
    awkward = [1.0, 1 - 2 ** -24, 1 - 2 ** -23, 0.5 + 2 ** -24, 0.75, 1e-6, 2 ** -40, 0.0]
    out = subprocess.run([exe, *(f"{b:.17g}" for b in corrections + awkward)], capture_output=True, text=True, check=True)
    assert not out.stdout, out.stdout


LAUNCHERS = r"""
extern "C" {
int pb_last_peer(const long* peers, int n, void* stream) { return (int)peers[n - 1] - (int)(long)stream; }
int pb_half(float x, void* stream) { return (int)(2 * x) - (int)(long)stream; }
int pb_is_null(const void* p, int n, void* stream) { return (p == nullptr) + 10 * n - (int)(long)stream; }
int pb_first_byte(const char* text) { return text[0]; }
int pb_next_peer(const long* peers, int n) { return (int)peers[n - 1] + 1; }
}
"""


@pytest.fixture
def launchers(tmp_path, monkeypatch):
    """A library of host functions in the place of the kernels' launchers; the current stream is 7."""
    lib = ctypes.CDLL(str(_compile(tmp_path, "launchers", LAUNCHERS, "-shared", "-fPIC")))
    monkeypatch.setattr(_lib, "_LIB", lib)
    monkeypatch.setattr(_lib, "_BOUND", {})
    monkeypatch.setattr(_lib, "LAUNCH_COUNT", 0)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 7)


def _table(*values):
    return (ctypes.c_long * len(values))(*values)


def test_launcher_takes_peer_tables_of_any_length(launchers):
    for n in (2, 8, 4):
        _lib.call("last_peer", _table(*range(n - 1), 7), n)
        assert _lib.call_ret("next_peer", _table(*range(n)), n) == n
    assert _lib.LAUNCH_COUNT == 3


@pytest.mark.parametrize("first,second", [((None, 0), (torch.zeros(1), 1)), ((torch.zeros(1), 1), (None, 0)),
                                          ((0, 0), (None, 0)), ((0, ctypes.c_int(0)), (torch.zeros(1), 1)),
                                          ((_table(1), 1), (None, ctypes.c_long(0)))])
def test_launcher_takes_other_kinds_than_on_its_first_call(launchers, first, second):
    """A null pointer (None or 0) and a tensor, plain and ctypes integers, in either order."""
    for _ in range(2):
        for p, n in (first, second):
            with pytest.raises(_lib.NativeLibraryError, match=f"code {-6 if not getattr(n, 'value', n) else 3}"):
                _lib.call("is_null", p, n)
    assert _lib.LAUNCH_COUNT == 4


def test_launcher_takes_floats_after_an_integer(launchers):
    with contextlib.suppress(_lib.NativeLibraryError):
        _lib.call("half", 1)             # (an integer in a float's place is not converted on the first call)
    _lib.call("half", 3.5)
    _lib.call("half", 3.5)
    assert _lib.call_ret("first_byte", b"a") == ord("a")


MIXED = r"""
extern "C" int pb_mixed(const void* a, int b, float c, long d, float e, const void* f, int g, int h, float i, long j, int k, int l,
                        float m, long n, int o, long p, void* stream) {
  return !(a == (void*)16 && b == -3 && c == 1.5f && d == -(1L << 40) && e == -0.25f && !f && g == 7 && h == -8 && i == 3.f &&
           j == 9 && k == 1 && l == 0 && m != m && n == 13 && o == -1 && p == (1L << 62) && stream == (void*)7);
}
extern "C" int pb_nine(float a, float b, float c, float d, float e, float f, float g, float h, float i, int n, void* stream) {
  return (int)(a + b + c + d + e + f + g + h + 2 * i) + n - (int)(long)stream;
}
"""


@pytest.mark.parametrize("compiled", [True, False])
def test_launcher_arguments_keep_their_places(compiled, tmp_path, monkeypatch):
    """Integers beyond the six registers between floats, 32-bit negatives, an integer in a float's place; more floats than
    registers.  Through the compiled binding and through ctypes."""
    if compiled and _lib._LAUNCH is None:
        pytest.skip("the binding is not built")
    monkeypatch.setattr(_lib, "_LIB", ctypes.CDLL(str(_compile(tmp_path, "mixed", MIXED, "-shared", "-fPIC"))))
    monkeypatch.setattr(_lib, "_BOUND", {})
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 7)
    if not compiled:
        monkeypatch.setattr(_lib, "_LAUNCH", None)
    for i in (3.0, 3):
        _lib.call("mixed", 16, -3, 1.5, -(1 << 40), -0.25, None, 7, -8, i, 9, True, False, float("nan"), 13, -1, 1 << 62)
    with pytest.raises(_lib.NativeLibraryError, match="code 1"):
        _lib.call("mixed", 16, -3, 1.5, -(1 << 40), -0.25, None, 7, -8, 4, 9, True, False, float("nan"), 13, -1, 1 << 62)
    _lib.call("nine", *[1.0] * 8, 2.0, -5)
    with pytest.raises(ctypes.ArgumentError):
        _lib.call("nine", *[1.0] * 8, object(), -5)


def test_binding_that_does_not_load_leaves_ctypes(tmp_path, monkeypatch):
    monkeypatch.setattr(_lib, "LIB_PATH", tmp_path / "library.so")
    assert _lib._load_launch() is None                                            # not built
    (tmp_path / build.LAUNCH_PATH.name).write_bytes(b"cut off")
    with pytest.warns(UserWarning, match="through ctypes"):
        assert _lib._load_launch() is None


@pytest.mark.parametrize("gcc", ["missing", "failing"])
def test_build_without_a_working_gcc_leaves_ctypes(gcc, tmp_path, monkeypatch, capsys):
    """The build goes on, and a binding of an older source is not left behind."""
    stale = tmp_path / "binding.so"
    stale.write_bytes(b"")
    monkeypatch.setattr(build, "LAUNCH_PATH", stale)
    monkeypatch.setenv("PATH", str(tmp_path))
    if gcc == "failing":
        (tmp_path / "gcc").write_text("#!/bin/sh\nexit 1\n")
        (tmp_path / "gcc").chmod(0o755)
    build._build_launch(force=True)
    assert not stale.exists() and "through ctypes" in capsys.readouterr().err


# Stands in for the CUDA runtime: launches are recorded as "device <d> shared <bytes>", and refused where a kernel asks for more
# than 48 KB without having been given the attribute on that device, or when `fail_next` says so.
RUNTIME = r"""
#include <cstdio>
#include <map>
#include <utility>
struct dim3_ { unsigned x, y, z; };
static int device, error, fail_next;
static std::map<std::pair<int, const void*>, int> limit;
static char log_[1 << 16];
static int used;
extern "C" {
void fake_device(int d) { device = d; }
void fake_fail_next(int n) { fail_next = n; }
const char* fake_log() { return log_; }
int cudaGetDevice(int* d) { *d = device; return 0; }
int cudaFuncSetAttribute(const void* f, int, int value) { limit[{device, f}] = value; return 0; }
int cudaGetLastError() { int e = error; error = 0; return e; }
int cudaLaunchKernel(const void* f, dim3_, dim3_, void**, size_t shared, void*) {
  used += snprintf(log_ + used, sizeof log_ - used, "device %d shared %zu\n", device, shared);
  if (shared > 48 * 1024 && (int)shared > limit[{device, f}]) error = 1;
  if (fail_next > 0 && --fail_next == 0) error = 700;
  return error;
}
struct Config { dim3_ grid, block; size_t shared; void *stream, *attrs; unsigned num_attrs; };
int cudaLaunchKernelExC(const Config* c, const void* f, void** args) {
  return cudaLaunchKernel(f, c->grid, c->block, args, c->shared, c->stream);
}
int cudaFree(void*) { return 0; }
int cudaDeviceGetAttribute(int* n, int, int) { *n = 148; return 0; }
int cudaOccupancyMaxActiveClusters(int* n, const void*, const void*) { *n = 74; return 0; }
static int encode() { return 0; }
int cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, int* status) { *f = (void*)encode; *status = 0; return 0; }
}
"""

BACKWARD = """
import ctypes, sys
fake = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)      # its names come before the runtime's
lib = ctypes.CDLL(sys.argv[2])
fake.fake_log.restype = ctypes.c_char_p
p, n = ctypes.c_void_p(4096), ctypes.c_long
rows, H, residual = int(sys.argv[3]), int(sys.argv[4]), int(sys.argv[5])
def backward():
    if H <= 256 and residual:                                 # norms of H-channel heads inside a packed tensor
        return lib.pb_qk_norm_bwd(p, p, p, p, p, p, p, p, p, n(rows), 2, 1, H, n(4 * H), n(4 * H), n(4 * H), 1, None)
    return lib.pb_rmsnorm_bwd(p, p, p, p, p if residual else None, p, p, p, n(rows), H, n(H), n(H), 1, None)
for step in sys.argv[6:]:
    what, value = step.split("=")
    if what == "device":
        fake.fake_device(int(value))
        print("rc", backward())
    else:
        fake.fake_fail_next(int(value))
print(fake.fake_log().decode())
"""


def _norm_backward(tmp_path, rows, H, residual, *steps):
    """Return codes and launches of RMSNorm backward calls on a stand-in for the CUDA runtime."""
    fake = _compile(tmp_path, "runtime", RUNTIME, "-shared", "-fPIC")
    out = subprocess.run([sys.executable, "-c", BACKWARD, fake, _lib.lib_path(), str(rows), str(H), str(int(residual)), *steps],
                         capture_output=True, text=True, check=True).stdout.split("\n")
    return [int(line.split()[1]) for line in out if line.startswith("rc")], [line for line in out if line.startswith("device")]


@pytest.mark.skipif(not _lib.available(), reason="the native library is not built")
@pytest.mark.parametrize("H", [1032, 2048, 4096, 8192, 16384])
@pytest.mark.parametrize("residual", [False, True])
def test_norm_backward_on_several_devices(tmp_path, H, residual):
    codes, launches = _norm_backward(tmp_path, 1000, H, residual, "device=0", "device=1", "device=0", "device=3")
    assert codes == [0, 0, 0, 0]
    assert [line.split()[1] for line in launches] == list("00110033")       # each the rows' kernel and the reduction


@pytest.mark.skipif(not _lib.available(), reason="the native library is not built")
@pytest.mark.parametrize("H", [64, 256, 512, 1024, 2048, 8192, 16384])
@pytest.mark.parametrize("residual", [False, True])
def test_norm_backward_stops_after_a_refused_launch(tmp_path, H, residual):
    """The weight gradient is not added up from partial sums that were never written."""
    codes, launches = _norm_backward(tmp_path, 1000, H, residual, "fail=1", "device=0", "device=0")
    assert codes == [700, 0] and len(launches) == 1 + (3 if H <= 256 and residual else 2)


NO_ROWS = """
import ctypes, sys
fake = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)
lib = ctypes.CDLL(sys.argv[2])
fake.fake_log.restype = ctypes.c_char_p
p, n = ctypes.c_void_p(4096), ctypes.c_long
for mode in (0, 2, 1):
    for H in (64, 4096):
        print(lib.pb_rmsnorm_bwd(p, p, p, p, p, p, p, p, n(0), H, n(H), n(H), mode, None),
              lib.pb_rmsnorm_bwd_two(None, None, p, None, None, None, None, p, p, n(0), H, n(H), n(H), mode, None), fake.fake_log().count(b"device"))
"""


@pytest.mark.skipif(not _lib.available(), reason="the native library is not built")
def test_norm_backward_of_no_rows_stores_the_gain_gradient(tmp_path):
    """Stored (fp32 or bf16): the reduction alone runs, and writes zeros.  Added: nothing runs.  Tensors of no rows have no
    address."""
    fake = _compile(tmp_path, "runtime", RUNTIME, "-shared", "-fPIC")
    out = subprocess.run([sys.executable, "-c", NO_ROWS, fake, _lib.lib_path()], capture_output=True, text=True, check=True).stdout
    assert out.split("\n")[:-1] == [f"0 0 {launches}" for launches in (2, 4, 6, 8, 8, 8)]


TENSOR_CORES = """
import ctypes, sys
fake = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)
lib = ctypes.CDLL(sys.argv[2])
p, n, f = ctypes.c_void_p(4096), ctypes.c_long, ctypes.c_float
def attention(d_qk, d_v, window, cap):
    sizes, q, k, v, o = (1, 256, 256, 0, 2, 2, d_qk, d_v), n(2 * d_qk), n(2 * d_qk), n(2 * d_v), n(2 * d_v)
    tail = (f(0.125), 1, window)
    return [lambda: lib.pb_flash_attn_fwd_cap(p, p, p, p, p, *sizes, q, k, v, o, *tail, None, f(cap), p, None),
            lambda: lib.pb_flash_attn_bwd_cap(*[p] * 10, *sizes, q, k, v, o, o, q, k, v, *tail, f(cap), p, None)]
calls = sum((attention(*d, w, c) for d in ((64, 64), (128, 128), (192, 128)) for w, c in ((0, 0.), (128, 0.), (0, 30.))), [])
for a_mn, b_mn in ((0, 0), (0, 1), (1, 1)):
    for out in (0, 1, 2):
        t = (512, 512, 512, n(512), n(512), n(512), a_mn, b_mn, out)
        calls += [lambda t=t: lib.pb_gemm_bf16(p, p, p, *t, 128, 0, p, None),
                  lambda t=t: lib.pb_gemm_bf16(p, p, p, *t, 256, 0, p, None),
                  lambda t=t: lib.pb_gemm_bf16_2cta(p, p, p, *t, 0, p, None),
                  lambda t=t: lib.pb_gemm_mxfp8(p, p, p, p, p, *t, 128, 0, p, None),
                  lambda t=t: lib.pb_gemm_mxfp8_2cta(p, p, p, p, p, *t, 0, p, None)]
for mode in (0, 1, 2):
    for e in (2, 256):
        for add in (0, 1):
            t = (mode, (256, 512, 512, e, p, p, p, add, p, None))
            calls += [lambda t=t: lib.pb_grouped_gemm(t[0], p, p, p, *t[1]),
                      lambda t=t: lib.pb_grouped_gemm_mxfp8(t[0], p, p, p, p, p, *t[1])]
calls += [lambda b=b: lib.pb_router_fwd(p, b, None, 64, 1024, 4, 0, 0, 1, 1, f(1), p, p, p, None, None) for b in (0, 1)]
first = [call() for call in calls]
for device in (1, 0, 3):
    fake.fake_device(device)
    assert [call() for call in calls] == first, device
print(len(calls), sum(rc == 0 for rc in first), sorted(set(first)))
"""


@pytest.mark.skipif(not _lib.available(), reason="the native library is not built")
def test_tensor_core_launchers_on_several_devices(tmp_path):
    """A kernel's shared-memory limit belongs to a device: what a launcher does on the first one it does on the others."""
    fake = _compile(tmp_path, "runtime", RUNTIME, "-shared", "-fPIC")
    out = subprocess.run([sys.executable, "-c", TENSOR_CORES, fake, _lib.lib_path()], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr
    total, launched = map(int, out.stdout.split()[:2])
    assert launched == total, out.stdout


@pytest.mark.parametrize("off,rows", [(0, 4), (1, 4), (3, 1), (8, 2)])
def test_gradient_of_packed_heads_is_read_from_an_aligned_start(off, rows):
    """The kernels read 16 bytes at a time: a contiguous view that starts in between is copied, any other is not."""
    g = torch.arange(off + rows * 64, dtype=torch.float32).bfloat16()[off:].view(rows, 64)
    got = fused.dense_rows(g)
    assert torch.equal(got, g) and got.is_contiguous() and got.data_ptr() % 16 == 0
    assert (got.data_ptr() == g.data_ptr()) == (g.data_ptr() % 16 == 0)
    wide = torch.arange(rows * 128, dtype=torch.float32).bfloat16().view(rows, 128)
    got = fused.dense_rows(wide[:, 8:72])
    assert torch.equal(got, wide[:, 8:72]) and got.is_contiguous() and got.data_ptr() % 16 == 0


def _norm_launchers(monkeypatch):
    """The norm kernels' launchers in plain PyTorch: every tensor is read and written by the row pitch that the launcher gets, from
    its own start; a pitch that leaves the tensor's memory raises, as does a start that 16-byte accesses cannot have."""
    def at(t, rows, H, pitch):
        assert t.data_ptr() % 16 == 0 and pitch % 8 == 0
        return torch.as_strided(t, (rows, H), (pitch, 1))

    def fwd(x, res, w, y, xsum, rstd, rows, H, ldx, ldy, eps):
        v = at(x, rows, H, ldx)
        if res is not None:
            v = at(xsum, rows, H, ldx).copy_(v.float() + at(res, rows, H, ldx).float())
        r = torch.rsqrt(v.float().pow(2).mean(1) + eps)
        if rstd is not None:
            rstd.copy_(r)
        at(y, rows, H, ldy).copy_(v.float() * r[:, None] * w.float())

    def bwd(dy, x, w, rstd, dres, dx, dx2, dw, rows, H, ldx, lddy):
        g, v, r = at(dy, rows, H, lddy).float(), at(x, rows, H, ldx).float(), rstd[:, None]
        d = r * g * w.float() - v * r ** 3 * (g * w.float() * v).mean(1, keepdim=True)
        if dres is not None:
            d = d + at(dres, rows, H, ldx).float()
        for out in (dx, dx2):
            if out is not None:
                at(out, rows, H, ldx).copy_(d)
        dw.copy_((g * v * r).sum(0))

    names = []

    def call(name, *a):
        names.append(name)
        if name == "rmsnorm_fwd":
            fwd(*a)
        elif name == "rmsnorm_bwd_two":
            bwd(*a[:8], *a[9:13])
        else:
            assert name == "rmsnorm_bwd"
            bwd(*a[:6], None, a[6], *a[8:12])

    monkeypatch.setattr(_lib, "call", call)
    monkeypatch.setattr(_lib, "call_ret", lambda name, rows: min(rows, 296))
    return names


@pytest.mark.parametrize("residual", [None, "dense", "same pitch", "other pitch"])
@pytest.mark.parametrize("where", ["columns", "rows", "every other row", "odd start", "one row for all"])
def test_norm_of_rows_with_a_pitch(monkeypatch, where, residual):
    """Inputs that are views: outputs and gradients are those of dense copies, and nothing outside the tensors is touched."""
    _norm_launchers(monkeypatch)
    g = torch.Generator().manual_seed(3)
    rows, H, W = 5, 16, 48

    def view(base):
        return {"columns": base[:rows, 8:8 + H], "rows": base.reshape(-1)[H:H + rows * H].view(rows, H),
                "every other row": base.reshape(-1, H)[:2 * rows:2], "odd start": base.reshape(-1)[4:4 + rows * H].view(rows, H),
                "one row for all": base[:1, :H].expand(rows, H)}[where]

    def wide():
        return torch.randn(rows, W, generator=g).bfloat16()

    x = view(wide())
    r = {None: None, "dense": torch.randn(rows, H, generator=g).bfloat16(), "same pitch": view(wide()),
         "other pitch": torch.randn(rows, 3 * H, generator=g).bfloat16()[:, H:2 * H]}[residual]
    dy, ds = (view(wide()) for _ in range(2))
    w = (1 + 0.1 * torch.randn(H, generator=g)).bfloat16()

    def run(*ts):
        x, r, dy, ds = (None if t is None else t.detach() for t in ts)
        p = torch.nn.Parameter(w.clone())
        x.requires_grad_()
        if r is None:
            y = fused.RMSNormFn.apply(x, p, 1e-5, None)
            y.backward(dy)
            return [y.detach(), x.grad, p.grad]
        r.requires_grad_()
        y, s = fused.RMSNormFn.apply(x, p, 1e-5, r)
        torch.autograd.backward([y, s], [dy, ds])
        return [y.detach(), s.detach(), x.grad, r.grad, p.grad]

    got = run(x, r, dy, ds)
    want = run(*(None if t is None else t.contiguous().clone() for t in (x, r, dy, ds)))
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def test_norm_gradient_is_written_twice_only_for_first_gradients_of_two_leaves(monkeypatch):
    """Elsewhere nothing copies the gradient that hidden and residual share, and a second store would be pure cost."""
    names = _norm_launchers(monkeypatch)
    g = torch.Generator().manual_seed(4)
    x, r, dy, ds = (torch.randn(3, 16, generator=g).bfloat16() for _ in range(4))
    w = torch.nn.Parameter(torch.ones(16, dtype=torch.bfloat16))
    x.requires_grad_(), r.requires_grad_()

    def last(step, a=x, b=r):
        out = fused.RMSNormFn.apply(a, w, 1e-5, b)
        got = step(out)
        return names[-1], got

    def backward(out):
        torch.autograd.backward(out, [dy, ds])

    assert last(backward)[0] == "rmsnorm_bwd_two"
    first = x.grad.clone()
    assert torch.equal(x.grad, r.grad) and x.grad.data_ptr() != r.grad.data_ptr()
    assert last(backward)[0] == "rmsnorm_bwd"
    assert torch.equal(x.grad, 2 * first) and torch.equal(r.grad, 2 * first)
    for only in (x, r):                       # one of the two has a gradient
        x.grad, r.grad = None, None
        only.grad = torch.zeros_like(x)
        assert last(backward)[0] == "rmsnorm_bwd"
        assert torch.equal(x.grad, first) and torch.equal(r.grad, first) and x.grad.data_ptr() != r.grad.data_ptr()
    x.grad = r.grad = None
    name, got = last(lambda out: torch.autograd.grad(out, [x, r], [dy, ds]))
    assert name == "rmsnorm_bwd" and torch.equal(got[0], first) and torch.equal(got[1], first)
    assert last(backward, x * 1)[0] == "rmsnorm_bwd" and torch.equal(x.grad, first) and torch.equal(r.grad, first)
    x.grad = r.grad = None
    assert last(backward, x, x)[0] == "rmsnorm_bwd"


@pytest.mark.parametrize("shape", [(6, 16), (2, 3, 16)])
@pytest.mark.parametrize("layer", [False, True])
@pytest.mark.parametrize("what", ["both", "first", "second"])
@pytest.mark.parametrize("leaves", ["both", "hidden", "residual"])
def test_leaves_of_a_norm_do_not_share_their_gradients_memory(monkeypatch, shape, layer, what, leaves):
    """Hidden and residual get the same gradient, each in memory of its own: a second pass doubles it, and one of them can be
    changed in place."""
    _norm_launchers(monkeypatch)
    g = torch.Generator().manual_seed(5)
    x, r, dy, ds = (torch.randn(*shape, generator=g).bfloat16() for _ in range(4))
    w = torch.nn.Parameter((1 + 0.1 * torch.randn(16, generator=g)).bfloat16())
    p = torch.nn.Parameter(torch.randn(16, 16, generator=g).bfloat16())

    def run():
        a, b = (t if leaves in ("both", name) else t.view_as(t) for t, name in ((x, "hidden"), (r, "residual")))
        out = layers.NormLinearFn.apply(a, b, w, p, 1e-5, None, False) if layer else fused.RMSNormFn.apply(a, w, 1e-5, b)
        pairs = list(zip(out, (dy.reshape(out[0].shape), ds)))
        torch.autograd.backward(*zip(*{"both": pairs, "first": pairs[:1], "second": pairs[1:]}[what]))

    x.requires_grad_(), r.requires_grad_()
    run()
    first = [t.grad.clone() for t in (x, r)]
    assert torch.equal(*first) and x.grad.data_ptr() != r.grad.data_ptr()
    run()
    assert torch.equal(x.grad, 2 * first[0]) and torch.equal(r.grad, 2 * first[1])
    x.grad.zero_()
    assert torch.equal(r.grad, 2 * first[1])


@pytest.mark.parametrize("sinks", [torch.zeros(2, dtype=torch.bfloat16), torch.zeros(3), torch.zeros(4)[::2]])
def test_attention_backward_refuses_sinks_the_kernel_cannot_read(sinks, monkeypatch):
    """The gradient kernel reads one contiguous fp32 logit per head, as the forward checks: nothing is launched for others."""
    q = torch.zeros(128, 2, 64, dtype=torch.bfloat16)
    launched = []
    monkeypatch.setattr(_lib, "call", lambda name, *args: launched.append(name))
    monkeypatch.setattr(_lib, "status_word", lambda device: None)
    with pytest.raises(AssertionError):
        attention.flash_attn_bwd(q, q, q, q, q, torch.zeros(1, 2, 128), 1, True, 0.125, sinks=sinks)
    assert not launched
    attention.flash_attn_bwd(q, q, q, q, q, torch.zeros(1, 2, 128), 1, True, 0.125, sinks=torch.zeros(2))
    assert launched == ["flash_attn_bwd_cap", "attn_sink_grad"]
