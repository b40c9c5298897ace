"""Arguments of a dependent launch are converted as those of an ordinary one: a pointer to another type does not compile."""
import shutil
import subprocess
from pathlib import Path

import pytest

from primus_b200 import build

KERNEL = r"""
#include "common.cuh"
__global__ void kern(float* out, const int* in, long n, float scale) { if (pb::grid_wait() && n) out[0] = in[0] * scale; }
int launch(%s* p, int* q, int n, cudaStream_t s) {
  pbh::launch_dependent(kern, 1, 32, 0, s, p, q, n, 2);
  return (int)cudaGetLastError();
}
"""


@pytest.mark.skipif(not (shutil.which("nvcc") or Path("/usr/local/cuda/bin/nvcc").exists()), reason="needs nvcc")
@pytest.mark.parametrize("pointer,compiles", [("float", True), ("double", False), ("void", False)])
def test_argument_types(tmp_path, pointer, compiles):
    (tmp_path / "k.cu").write_text(KERNEL % pointer)
    cmd = [build.find_nvcc(), *build.NVCC_FLAGS, "-I", str(build.CSRC), "-c", str(tmp_path / "k.cu"), "-o", str(tmp_path / "k.o")]
    p = subprocess.run(cmd, capture_output=True, text=True)
    assert (p.returncode == 0) == compiles, p.stderr
