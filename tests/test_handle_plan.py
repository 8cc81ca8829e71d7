"""CPU check of a handle's device memory (tests/cpp/handle_plan_check.cu): one allocation per handle, sized
by the buffers that the handle then takes from it, and a serving request counted with all of them. Host code linked with the library's objects and a CUDA
runtime that only counts; no GPU needed."""
import glob
import os
import shutil
import subprocess

import pytest

from opentm_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)


@pytest.mark.skipif(NVCC is None, reason="needs nvcc")
def test_handle_memory(tmp_path):
    build.build()  # the library's objects, where they are not there yet
    exe = tmp_path / "handle_plan_check"
    subprocess.run([NVCC, *build.host_compiler(), *build.ARCH, "-std=c++17", "-O1", "--expt-relaxed-constexpr",
                    "-cudart", "none", "-I", os.path.join(ROOT, "include"), "-I", build.CSRC,
                    "-Xlinker", "--unresolved-symbols=ignore-all",
                    *(os.path.join(ROOT, "tests", "cpp", f) for f in ("handle_plan_check.cu", "counting_runtime.cpp")),
                    *sorted(glob.glob(os.path.join(build.BUILD_DIR, "*.o"))), "-o", str(exe)], check=True, timeout=600)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.strip() == "ok"
