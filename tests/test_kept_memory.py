"""Device memory that a context keeps between calls: its ownership rules, run on
the host against a counting stand-in for the device allocator, and that every
allocation of a context can have it back."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "voreen_gb300", "csrc")


def test_ownership_on_a_counting_allocator(tmp_path):
    from voreen_gb300 import build
    cc, inc = shutil.which("g++"), os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    if cc is None or not os.path.exists(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path / "kept_memory")
    subprocess.run([cc, "-std=c++17", "-Wall", "-O1", "-UNDEBUG", "-I", inc, os.path.join(ROOT, "tests", "native", "kept_memory.cpp"),
                    os.path.join(CSRC, "kept.cpp"), "-pthread", "-o", exe], check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "kept_memory ok" in r.stdout, r.stderr + r.stdout


def test_allocations_of_a_context_go_through_device_alloc():
    """Plain cudaMalloc: device_alloc itself, a context's first allocations
    (nothing is kept yet), the processor's images (which trim and try again)
    and the volume generator, which has no context."""
    plain = {}
    for f in sorted(os.listdir(CSRC)):
        src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read()) if f.endswith((".cpp", ".cu", ".cuh", ".h")) else ""
        n = len(re.findall(r"\bcudaMalloc\(", src))
        if n:
            plain[f] = n
    assert plain == {"kept.cpp": 2, "api.cpp": 2, "processor.cpp": 2, "synth_tubes.cu": 1}
    src = open(os.path.join(CSRC, "api.cpp")).read()
    create = src[src.index("vrc_status vrc_context_create("):src.index("vrc_status vrc_context_destroy(")]
    assert len(re.findall(r"\bcudaMalloc\(", create)) == 2
