"""Device allocations (csrc/device_mem.h): one that fails for want of memory is
tried once more after the pools gave back what they cache, any other result
stands. Against fakes of the allocator, compiled here; no GPU needed."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "oxideav-render_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "device_mem.h"
// Results of the fake allocator's first and second call -> what the caller
// gets, how often it was called, and whether the trim came between.
static void one(cudaError_t first, cudaError_t second) {
  int calls = 0, trims = 0, trims_before_second = -1;
  const cudaError_t e = ptd::alloc_or_trim(
      [&] {
        if (++calls == 2) trims_before_second = trims;
        return calls == 1 ? first : second;
      },
      [&] { ++trims; });
  std::printf("%d %d %d %d\n", (int)e, calls, trims, trims_before_second);
}
int main() {
  one(cudaSuccess, cudaErrorUnknown);
  one(cudaErrorMemoryAllocation, cudaSuccess);
  one(cudaErrorMemoryAllocation, cudaErrorMemoryAllocation);
  one(cudaErrorMemoryAllocation, cudaErrorInvalidValue);
  one(cudaErrorInvalidValue, cudaSuccess);
  std::printf("%d %d\n", (int)cudaErrorMemoryAllocation, (int)cudaErrorInvalidValue);
}
"""


def cuda_include():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(cuda_include()), reason="no g++ or CUDA headers")
def test_a_failed_allocation_is_tried_again_after_a_trim(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-I", cuda_include(), str(src), "-o", str(exe)], check=True)
    rows = [tuple(map(int, l.split())) for l in
            subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()]
    oom, invalid = rows.pop()
    assert rows == [(0, 1, 0, -1), (0, 2, 1, 1), (oom, 2, 1, 1), (invalid, 2, 1, 1), (invalid, 1, 0, -1)]
