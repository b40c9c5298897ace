"""Host-side parts of the native library, on a machine without a GPU."""
import subprocess
from pathlib import Path

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
