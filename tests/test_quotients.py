"""The written-out divisions of the device arithmetic on the host (no GPU):
over_light_speed and divide3 give the IEEE quotients bit for bit, whatever
their operands.  tests/quotient_check.cu, compiled for the host with nvcc."""
import subprocess
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "corsika8-kokkos_b200" / "csrc"


def test_written_out_divisions_are_the_ieee_quotients(tmp_path):
    out = tmp_path / "quotient_check"
    cmd = ["/usr/local/cuda/bin/nvcc", "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a",
           "-Xcompiler", "-ffp-contract=off", "-I", str(CSRC), "-x", "cu", str(HERE / "quotient_check.cu"),
           "-o", str(out)]
    built = subprocess.run(cmd, capture_output=True, text=True, timeout=600)
    assert built.returncode == 0, built.stderr
    run = subprocess.run([str(out)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0 and run.stdout.strip() == "ok", run.stdout + run.stderr
