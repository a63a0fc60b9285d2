"""Which points a step reads where they lie: only aligned device memory of the
context's own GPU; all other memory that it accepts is copied first.  Host rule,
compiled with the host compiler; no GPU needed."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "glint_pipeline_gb300", "csrc")
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

pytestmark = pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA_INC),
                                reason="g++ or the CUDA headers not available")

SOURCE = r"""
#include <cstdio>
#include "step_points.h"
int main() {
    const cudaMemoryType types[] = {cudaMemoryTypeUnregistered, cudaMemoryTypeHost, cudaMemoryTypeDevice,
                                    cudaMemoryTypeManaged};
    for (int t = 0; t < 4; ++t)
        for (int device = 0; device < 2; ++device)
            for (int off = 0; off < 16; off += 8) {
                cudaPointerAttributes at = {};
                at.type = types[t];
                at.device = device;
                const bool in = glint::points_in_place(at, 0, reinterpret_cast<void *>(0x10000 + off));
                if (in != (types[t] == cudaMemoryTypeDevice && device == 0 && off == 0)) {
                    std::printf("type %d device %d offset %d: %d\n", t, device, off, (int)in);
                    return 1;
                }
            }
    return 0;
}
"""


def test_only_own_aligned_device_memory_is_read_in_place(tmp_path):
    src, exe = tmp_path / "points.cpp", tmp_path / "points"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-I", CUDA_INC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
