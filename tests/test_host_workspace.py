"""The device memory that host-buffer calls keep, on the CPU: csrc/host_workspace.cu against a made-up
device (tests/cpp/host_workspace_check.cpp) that runs out of memory and whose contexts are destroyed."""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    if shutil.which("g++") is None or not (CUDA / "include" / "cuda_runtime_api.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    exe = tmp_path_factory.mktemp("host_workspace") / "check"
    env = {k: v for k, v in os.environ.items() if k not in ("CC", "CXX")}
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", str(CUDA / "include"), "-x", "c++",
                    str(ROOT / "cogni_ml_b200" / "csrc" / "host_workspace.cu"),
                    str(ROOT / "tests" / "cpp" / "host_workspace_check.cpp"), "-o", str(exe)],
                   check=True, env=env, capture_output=True, text=True)
    return exe


@pytest.mark.parametrize("what", ["memory", "contexts", "thread"])
def test_kept_blocks(check, what):
    out = subprocess.run([str(check), what], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
