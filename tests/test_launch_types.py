"""launch_chained (csrc/launch.h) converts its arguments as a call does: a
pointer of another type is an error when it is compiled, not a kernel reading
floats as doubles."""
import os
import subprocess

import pytest

from stzpp_gb300 import build

SOURCE = """
#include "launch.h"
__global__ void kernel(int n, const double *in, double *out) { stzmg::chain_wait(); if (n) out[0] = in[0]; }
void launch(%s *in, double *out) { stzmg::launch_chained(kernel, dim3(1), dim3(1), 0, nullptr, 1, 2u, in, out); }
void none(double *in) { stzmg::launch_chained(kernel, dim3(1), dim3(1), 0, nullptr, 1, 0, in, nullptr); }
"""


@pytest.mark.parametrize("held,compiles", [("double", True), ("const double", True), ("float", False), ("void", False)])
def test_pointer_types(held, compiles, tmp_path):
    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    src = tmp_path / "types.cu"
    src.write_text(SOURCE % held)
    flags = [f for f in build._flags() if f not in ("-O3", "-lineinfo")]
    r = subprocess.run([nvcc, *flags, "-O0", "-I", build.CSRC, "-c", str(src), "-o", os.devnull], capture_output=True,
                       text=True)
    assert (r.returncode == 0) == compiles, r.stderr[-600:]
