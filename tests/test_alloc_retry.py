"""An allocation of the library's that fails for want of memory is made again once
the scratch pool has given back what it keeps (a host program against the
header, the allocation faked); any other answer stands.
"""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "medimage_gb300", "csrc")
CUDA = "/usr/local/cuda/include"

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "alloc_retry.h"
int main() {
  int bad = 0;
  auto run = [&](std::vector<cudaError_t> answers, cudaError_t want, unsigned allocs, int given, const char *what) {
    unsigned calls = 0;
    int back = 0;
    const cudaError_t e = medimg::alloc_or_give_back([&] { return answers[calls++]; }, [&] { back++; });
    if (e != want || calls != allocs || back != given) std::printf("%s\n", what), bad++;
  };
  run({cudaSuccess}, cudaSuccess, 1, 0, "memory at once");
  run({cudaErrorMemoryAllocation, cudaSuccess}, cudaSuccess, 2, 1, "memory once it is given back");
  run({cudaErrorMemoryAllocation, cudaErrorMemoryAllocation}, cudaErrorMemoryAllocation, 2, 1, "none at all");
  run({cudaErrorInvalidValue}, cudaErrorInvalidValue, 1, 0, "another error");
  return bad;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA), reason="needs g++ and CUDA's headers")
def test_retry(tmp_path):
    src, exe = tmp_path / "retry.cpp", tmp_path / "retry"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-I", CUDA, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_every_allocation_goes_through_it():
    """One plain cudaMalloc in the library: the one that is repeated."""
    text = "".join(open(os.path.join(CSRC, f)).read() for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh", ".h")))
    assert len(re.findall(r"\bcudaMalloc\(", text)) == 1


@pytest.mark.gpu
def test_trim_gives_back(engine):
    """A projection of 3000^2 leaves its scratch (72 MB) in the pool; trimming
    hands it to the device, and the next projection is the same."""
    import numpy as np
    import torch

    p = engine.Plan.fan(engine.FanGeometry.covering(3000, 0.1, 8, 600))
    img = torch.tensor(np.random.default_rng(0).random(p.img_shape, dtype=np.float32), device="cuda")
    outs = [torch.empty(p.sino_shape, device="cuda") for _ in range(2)]
    engine.engine._check("trim", engine.lib().at_scratch_trim())
    p.forward_dev(img.data_ptr(), outs[0].data_ptr(), None)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    engine.engine._check("trim", engine.lib().at_scratch_trim())
    assert torch.cuda.mem_get_info()[0] - before >= 2 * 3000 * 3000 * 4
    p.forward_dev(img.data_ptr(), outs[1].data_ptr(), None)
    torch.cuda.synchronize()
    assert torch.equal(outs[0], outs[1])
