"""Offsets into the ket tables at the sizes that context creation admits (2^32
doubles in all; any number of positions an int holds): compiled and compared on
the CPU."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "iqcp_b200", "csrc")
CODE = """
#include "engine.cuh"
using namespace iqcp;
constexpr bool fits(int np) {  // the last field of a bucket's last primitive and ket; one more ket would not fit
  return 8LL * np * max_bucket_kets(np) <= 0x7fffffffLL && 8LL * np * (max_bucket_kets(np) + 1LL) > 0x7fffffffLL;
}
static_assert(fits(1) && fits(3) && fits(36) && fits(1296) && max_bucket_kets(0) == max_bucket_kets(1), "one bucket");
static_assert(max_bucket_kets((1 << 28) - 1) == 1 && max_bucket_kets(1 << 28) == 0, "longest ket");
static_assert(ket_geom_offset(6, 400000000) == 2400000000LL, "positions");
"""


def test_offsets_beyond_an_int(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    src = tmp_path / "offsets.cu"
    src.write_text(CODE)
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-I", CSRC, "-c", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-o", str(tmp_path / "offsets.o"), str(src)], check=True)
