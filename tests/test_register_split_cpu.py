"""A warpgroup that asks for more registers than the block was launched with waits for good: the prompt attention's two shares have
to add up to no more than what the compiler gives its threads at launch."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
def test_the_shares_of_the_warpgroups_fit_the_launch(tmp_path):
    csrc = os.path.join(ROOT, "async-gpu_b200", "csrc")
    with open(os.path.join(csrc, "attention_tc.cu")) as f:
        source = f.read()
    shares = [int(n) for n in re.findall(r"setmaxnreg\.(?:inc|dec)\.sync\.aligned\.u32 (\d+)", source)]
    threads = int(re.search(r"NTHREADS = (\d+)", source).group(1))
    assert len(shares) == 2 and threads == 128 * len(shares)
    r = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-I", os.path.join(ROOT, "include"), "-I", csrc,
                        "-Xptxas", "-v", "-c", os.path.join(csrc, "attention_tc.cu"), "-o", str(tmp_path / "attention.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    used = re.search(r"prefill_attn_tc_kernel.*?Used (\d+) registers", r.stderr, re.S)
    assert 128 * sum(shares) <= threads * int(used.group(1))
    assert 2 * threads * int(used.group(1)) <= 65536  # two blocks per SM
    assert "0 bytes spill stores" in r.stderr
