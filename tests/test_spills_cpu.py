"""The GEMVs of few rows hold their weights in registers across the wait on the kernel before them; values that the compiler
has to spill there go to local memory and back in every step (up to 400 bytes of a thread once did)."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
@pytest.mark.parametrize("source", ["int4_gemv.cu", "linear_f32.cu"])
def test_gemvs_keep_their_values_in_registers(tmp_path, source):
    csrc = os.path.join(ROOT, "async-gpu_b200", "csrc")
    r = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-I", os.path.join(ROOT, "include"), "-I", csrc,
                        "-Xptxas", "-v", "-c", os.path.join(csrc, source), "-o", str(tmp_path / "gemv.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    spilled = {m[0]: int(m[1]) for m in re.findall(r"Compiling entry function '(\S+)'(?:(?!Compiling).)*?(\d+) bytes spill stores", r.stderr, re.S)}
    assert len(spilled) > 4
    assert not {k: v for k, v in spilled.items() if "gemv" in k and v > 16}  # 16: two pointers before the loop
