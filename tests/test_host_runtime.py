"""The runtime's buffer pools on the CPU, against a CUDA runtime whose streams run when they are waited for
(tests/host_runtime_probe.cpp): a block may not be handed out while work that uses it is in flight, whatever
another thread does meanwhile."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "minilake_b200", "csrc")


def test_blocks_in_use_are_not_handed_out(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    exe = str(tmp_path / "host_runtime_probe")
    subprocess.run(["g++", "-std=c++17", "-O0", "-I", CSRC, "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "host_runtime_probe.cpp"), os.path.join(CSRC, "ml_runtime.cpp"),
                    "-lpthread", "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0 and "FAILED" not in out.stdout, out.stdout + out.stderr
