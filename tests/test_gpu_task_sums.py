"""Sums of the task counts: whole where they fit an int, refused where they do not,
whatever the sums of single chunks wrap to."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu
CSRC = os.path.join(ROOT, "iqcp_b200", "csrc")
CODE = """
#include "tasks.cu"
#include <cstdio>
#include <vector>
using namespace iqcp;

// offsets of n counts, as launch_task_offsets chains the kernels
template <typename N, typename P>
int check(void (*chunk)(N, int*, P*), void (*parts)(int, P*), void (*add)(N, int, int*, const P*), int n, int each, long long want) {
  const int chunks = (n + 1023) / 1024;
  std::vector<int> h(n + 1, each);
  int* v;
  P* part;
  if (cudaMalloc(&v, sizeof(int) * (n + 1)) != cudaSuccess || cudaMalloc(&part, sizeof(P) * (chunks + 1)) != cudaSuccess) return 1;
  cudaMemcpy(v, h.data(), sizeof(int) * n, cudaMemcpyHostToDevice);
  chunk<<<chunks, 1024>>>(n, v, part);
  parts<<<1, 1024>>>(chunks, part);
  add<<<chunks, 1024>>>(n, chunks, v, part);
  cudaMemcpy(h.data(), v, sizeof(int) * (n + 1), cudaMemcpyDeviceToHost);
  cudaFree(v);
  cudaFree(part);
  bool ok = cudaGetLastError() == cudaSuccess && h[n] == want;
  for (int i = 0; ok && want >= 0 && i < n; ++i) ok = h[i] == (long long)i * each;
  if (!ok) std::printf("n %d each %d: total %d, not %lld\\n", n, each, h[n], want);
  return !ok;
}

int main() {
  int bad = 0;
  const auto run = [&](int n, int each, long long want) {
    bad += check(scan_chunks_kernel, scan_parts_kernel, scan_add_kernel, n, each, want);
  };
  run(1, 7, 7);
  run(1023, 3, 3069);
  run(1024, 3, 3072);
  run(1025, 3, 3075);
  run(1024 * 1024 + 5, 2000, 2000LL * (1024 * 1024 + 5));  // 1025 chunks, just below 2^31
  run(2, 0x3fffffff, 0x7ffffffe);
  run(2048, 1 << 20, -1);                                  // 2^31: one too many
  run(4096, 1 << 22, -1);                                  // chunk sums of 2^32 wrap to nothing
  run(3000, 1 << 30, -1);
  return bad;
}
"""


def test_sums_beyond_an_int(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    src = tmp_path / "sums.cu"
    src.write_text(CODE)
    exe = str(tmp_path / "sums")
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-I", CSRC, "-gencode",
                    "arch=compute_100a,code=sm_100a", "-o", exe, str(src)], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
