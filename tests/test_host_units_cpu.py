"""Host-side parts of the library that need no GPU, compiled with g++ and run here (tests/cpp/*_test.cpp)."""
import subprocess
from pathlib import Path

import pytest

CPP = Path(__file__).resolve().parent / "cpp"


@pytest.mark.parametrize("name", ["once_per_device_test", "exp_of_gap_test"])
def test_unit(name, tmp_path):
    binary = tmp_path / name
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", str(CPP / (name + ".cpp")), "-o", str(binary)], check=True)
    out = subprocess.run([str(binary)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
