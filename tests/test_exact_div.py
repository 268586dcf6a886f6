"""The FP64 quotients and square roots that Euler forms on the integer pipe
(csrc/exact_int.h) give the bits of the IEEE operations: the same header,
compiled for the host, against the host's division and square root on random
operands, rounding boundaries and special values, with the seeds of the
device's approximation instructions moved by more than their documented error."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


def test_integer_pipe_quotients_and_roots_round_like_ieee(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "exact_div_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", str(exe), str(HERE / "exact_div_check.cpp")], check=True)
    out = subprocess.run([str(exe), "100000"], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "differ 0" in out.stdout
