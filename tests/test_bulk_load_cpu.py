"""bulk_load (csrc/tcgen05.cuh) copies whole pieces of 16 KB: a size that is not a
multiple would write past its place and never complete its barrier, so it does not
compile."""
import os
import subprocess

import pytest

from qcs_gb300 import build as B

SOURCE = """
#include "tcgen05.cuh"
__global__ void k(const void *src) {
  extern __shared__ __align__(16) unsigned char smem[];
  qcs::bulk_load<%d>(qcs::smem_u32(smem), src, qcs::smem_u32(smem));
}
"""


@pytest.mark.parametrize("size,compiles", [(16384, True), (131072, True), (8192, False),
                                           (16384 + 16, False)])
def test_sizes_of_bulk_copies(tmp_path, size, compiles):
    src = os.path.join(tmp_path, "bulk.cu")
    with open(src, "w") as f:
        f.write(SOURCE % size)
    p = subprocess.run([B.nvcc(), *B.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-c", src,
                        "-o", os.path.join(tmp_path, "bulk.o"), "-I", B.CSRC, "-I", B.INCLUDE],
                       capture_output=True, text=True)
    assert (p.returncode == 0) == compiles, p.stderr
    assert compiles or "whole pieces" in p.stderr
