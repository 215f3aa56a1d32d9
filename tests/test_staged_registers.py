"""The staged z pass in FP64 leaves the registers for two CTAs per SM.

A CTA has 256 threads and an SM 65,536 registers, so two of them fit while a
thread takes at most 128; the tile's share of the shared memory is chosen for
two.  The count is the compiler's own report for a translation unit that
instantiates the kernel alone (no GPU needed)."""
import os
import re
import subprocess

import pytest

from pyspectral_b200 import build as B

SRC = """
#include "psb_physics.cuh"
template __global__ void psb::zpass_kernel<double, psb::%s<double>, false>(psb::ZArgs<double>, psb::%s<double>);
"""


@pytest.mark.parametrize("phys", ["PhysProducts", "PhysSmag", "PhysMHD"])
def test_staged_z_pass_fp64_fits_two_ctas_per_sm(phys, tmp_path):
    cu = tmp_path / "z.cu"
    cu.write_text(SRC % (phys, phys))
    cmd = [B.nvcc()] + B.FLAGS + ["-I", B.CSRC, "-Xptxas", "-v", "-c", str(cu), "-o", os.devnull]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    used = [int(n) for n in re.findall(r"Used (\d+) registers", r.stdout + r.stderr)]
    assert used and max(used) <= 128, used
