"""raise_dyn_smem from two host threads: the limit ends at the larger of the
two requests, whichever thread looks first.  The factorisations raise their
kernel's limit on every call, so chains of different sizes on threads of their
own meet here; the CUDA calls are fakes."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = "/usr/local/cuda/include"

SOURCE = r"""
#include <chrono>
#include <thread>
#include "common.cuh"
static std::atomic<int> limit{0}, looks{0}, sets{0};
// the first caller looks at the limit and is then held until the other has set it (or half a second)
cudaError_t CUDARTAPI cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  a->maxDynamicSharedSizeBytes = limit;
  if (looks++ == 0)
    for (int k = 0; k < 500 && !sets; ++k) std::this_thread::sleep_for(std::chrono::milliseconds(1));
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaFuncSetAttribute(const void*, cudaFuncAttribute, int v) {
  limit = v;
  ++sets;
  return cudaSuccess;
}
static void kernel() {}
int main() {
  std::thread a([] { raise_dyn_smem(kernel, 100000); });
  while (!looks) std::this_thread::yield();
  std::thread b([] { raise_dyn_smem(kernel, 200000); });
  a.join();
  b.join();
  printf("%d\n", limit.load());
}
"""


@pytest.mark.skipif(not os.path.isdir(CUDA) or not shutil.which("g++"), reason="needs the CUDA headers and g++")
def test_two_threads_never_lower_the_limit(tmp_path):
    src, exe = tmp_path / "limit.cpp", tmp_path / "limit"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-w", "-O1", "-pthread", "-I", CUDA, "-I", os.path.join(ROOT, "pqmc_allinone_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True, timeout=120)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=30)
    assert r.stdout.strip() == "200000", r.stdout
