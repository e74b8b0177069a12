"""A kernel's opt-in to large shared memory holds for one device: another device
of the same process gets a call of its own, and a call that failed is repeated
(a host program against the header, the device and the call faked).
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = "/usr/local/cuda/include"

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "smem_optin.h"
int main() {
  medimg::SmemOptIn optin;
  int device = 0;
  cudaError_t answer = cudaSuccess;
  std::vector<std::pair<int, size_t>> calls;
  auto ensure = [&](int dev, size_t bytes) {
    device = dev;
    return optin.ensure(bytes, [&](int *d) { *d = device; return cudaSuccess; },
                        [&](size_t b) { calls.push_back({device, b}); return answer; });
  };
  int bad = 0;
  auto check = [&](bool ok, const char *what) { if (!ok) { std::printf("%s\n", what); bad++; } };
  check(ensure(0, 48 * 1024) == cudaSuccess && calls.empty(), "48 KB need no call");
  check(ensure(0, 66000) == cudaSuccess && calls.size() == 1, "the first call");
  check(ensure(0, 66000) == cudaSuccess && ensure(0, 50000) == cudaSuccess && calls.size() == 1, "one call a device");
  check(ensure(1, 66000) == cudaSuccess && calls.size() == 2 && calls[1].first == 1, "another device");
  check(ensure(0, 70000) == cudaSuccess && calls.size() == 3 && calls[2].second == 70000, "a larger size");
  answer = cudaErrorInvalidValue;
  check(ensure(2, 66000) == cudaErrorInvalidValue && calls.size() == 4, "an error is reported");
  answer = cudaSuccess;
  check(ensure(2, 66000) == cudaSuccess && calls.size() == 5, "and not kept");
  check(ensure(99, 66000) == cudaSuccess && ensure(99, 66000) == cudaSuccess && calls.size() == 7, "devices past the table");
  check(optin.ensure(66000, [](int *) { return cudaErrorNoDevice; }, [](size_t) { return cudaSuccess; }) ==
            cudaErrorNoDevice, "no device");
  return bad;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA), reason="needs g++ and CUDA's headers")
def test_opt_in_per_device(tmp_path):
    src, exe = tmp_path / "optin.cpp", tmp_path / "optin"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "medimage_gb300", "csrc"), "-I", CUDA,
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_no_launch_opts_in_past_it():
    """Every opt-in of the library goes through it."""
    csrc = os.path.join(ROOT, "medimage_gb300", "csrc")
    for name in sorted(os.listdir(csrc)):
        if name.endswith((".cu", ".cuh", ".cpp")):
            text = open(os.path.join(csrc, name)).read()
            assert text.count("cudaFuncAttributeMaxDynamicSharedMemorySize") == text.count("optin.ensure("), name
