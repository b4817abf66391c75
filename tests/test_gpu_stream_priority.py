"""A context's own side streams (the tree build's larger node classes) have the priority of the stream
its caller gave it.  The streams are internal, so a small host program reads them from the context."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "common.cuh"
int main() {
  int least, greatest;
  cudaDeviceGetStreamPriorityRange(&least, &greatest);
  for (int want = least; want >= greatest; want--) {
    cudaStream_t s;
    cudaStreamCreateWithPriority(&s, cudaStreamNonBlocking, want);
    bit_ctx_opts o{0, s, 0};
    bit_ctx* c = nullptr;
    if (bit_ctx_create(&c, &o)) return 2;
    const int n = 50000;  // several node classes
    std::vector<double> x[3];
    unsigned r = 1;
    for (auto& v : x)
      for (int i = 0; i < n; i++) v.push_back((r = r * 1664525u + 1013904223u) / 4294967296.0);
    bit_tree* t = nullptr;
    if (bit_tree_build(c, n, x[0].data(), x[1].data(), x[2].data(), 200, &t)) return 3;
    int made = 0;
    for (cudaStream_t side : c->c.side) {
      if (!side) continue;
      int p = 99;
      cudaStreamGetPriority(side, &p);
      made++;
      if (p != want) std::printf("side stream at %d, the context's at %d\n", p, want);
    }
    std::printf("priority %d: %d side streams\n", want, made);
    if (!made) return 4;
    bit_tree_destroy(t);
    bit_ctx_destroy(c);
    cudaStreamDestroy(s);
  }
  return 0;
}
"""


def test_side_streams_have_the_callers_priority(tmp_path):
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    if not shutil.which(nvcc):
        pytest.skip("no CUDA compiler")
    src, exe = tmp_path / "prio.cu", tmp_path / "prio"
    src.write_text(PROGRAM)
    lib = os.path.join(ROOT, "bit_b200", "lib")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-o", str(exe), str(src),
                    "-I", os.path.join(ROOT, "bit_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    "-L", lib, "-lbit_b200", "-Xlinker", "-rpath", "-Xlinker", lib], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out
    assert "priority -" in out.stdout and "side stream at" not in out.stdout, out.stdout
