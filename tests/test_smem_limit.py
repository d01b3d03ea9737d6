"""A kernel's shared-memory limit is raised once on every device that launches it."""
import glob
import os
import re
import shutil
import subprocess

import pytest

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tsplit_b200", "csrc", "kernels")

#: the three runtime names that the header uses, with a current device and a log of the calls
RUNTIME = """
#pragma once
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1 };
enum cudaFuncAttribute { cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
extern int device, fail, calls;
inline cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
template <class K> cudaError_t cudaFuncSetAttribute(K*, cudaFuncAttribute, int) {
  ++calls;
  return fail ? cudaErrorInvalidValue : cudaSuccess;
}
"""
PROGRAM = """
#include "smem_limit.h"
#include <cstdio>
int device = 0, fail = 0, calls = 0;
void one() {}
void two() {}
int main() {
  tsb_launch::SmemLimit a, b;
  const int on[] = {0, 0, 1, 0, 1, 63, 63, 64, 64};
  for (int d : on) { device = d; if (a.raise(one, 1 << 16) != cudaSuccess) return 2; std::printf("%d ", calls); }
  device = 5;
  fail = 1; if (b.raise(two, 1 << 16) == cudaSuccess) return 3;          // a refusal is not remembered as done
  fail = 0; if (b.raise(two, 1 << 16) != cudaSuccess) return 4;
  std::printf("%d", calls);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_limit_is_raised_per_device(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cc").write_text(PROGRAM)
    exe = tmp_path / "main"
    subprocess.run(["g++", "-std=c++17", "-I", str(tmp_path), "-I", KERNELS, str(tmp_path / "main.cc"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, stdout=subprocess.PIPE, text=True).stdout
    # first use of 0, 1 and 63; every use of 64; two tries of the second kernel
    assert [int(v) for v in out.split()] == [1, 1, 2, 2, 2, 3, 3, 4, 5, 7]


def test_launches_do_not_remember_it_per_process():
    for path in glob.glob(os.path.join(KERNELS, "*.cu")):
        text = open(path).read()
        for at in re.finditer(r"cudaFuncSetAttribute", text):
            before = text[max(0, at.start() - 200):at.start()]
            assert not re.search(r"static bool", before), os.path.basename(path)
