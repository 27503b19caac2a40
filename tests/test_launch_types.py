"""launch_behind takes arguments only as the kernel's parameters would take them: two pointers in
each other's place do not compile, as with a launch in angle brackets."""
import os
import subprocess

import pytest

from cosmictiger_b200 import build as b

SOURCE = """
#include "ct_internal.cuh"
__global__ void k(int64_t n, const float* a, int* i) { i[n] = a[n] > 0.f; }
cudaError_t launch(cudaStream_t st, int n, float* a, int* i) { return ct::launch_behind(k, 1, 32, st, n, %s); }
"""


@pytest.mark.parametrize("args,compiles", [("a, i", True), ("i, i", False), ("a, a", False)])
def test_swapped_pointers_do_not_compile(tmp_path, args, compiles):
    if not os.path.exists(b.NVCC):
        pytest.skip("nvcc not installed")
    src = tmp_path / "launch.cu"
    src.write_text(SOURCE % args)
    r = subprocess.run([b.NVCC] + b.ARCH + b.COMMON + ["-c", str(src), "-o", str(tmp_path / "launch.o")], capture_output=True, text=True)
    assert (r.returncode == 0) == compiles, r.stderr
