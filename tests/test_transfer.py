"""The result copies (transfer.hpp) on the host against a CUDA runtime of the
test's own (no GPU): tests/ring_check.cpp, compiled with g++."""
import subprocess
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "corsika8-kokkos_b200" / "csrc"


def test_result_copies_on_a_host_runtime(tmp_path):
    out = tmp_path / "ring_check"
    cmd = ["g++", "-std=c++17", "-O1", "-Wall", "-pthread", "-I", str(CSRC), "-I", "/usr/local/cuda/include",
           str(HERE / "ring_check.cpp"), "-o", str(out)]
    built = subprocess.run(cmd, capture_output=True, text=True, timeout=300)
    assert built.returncode == 0, built.stderr
    run = subprocess.run([str(out)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0 and run.stdout.strip() == "ok", run.stdout + run.stderr
