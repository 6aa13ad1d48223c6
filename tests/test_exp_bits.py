"""The conversions between double and float by bit patterns against the compiler's."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_conversions_by_bits_are_the_conversions(tmp_path):
    exe = tmp_path / "exp_bits_check"
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{ROOT}/viennaemc_gb300/csrc",
                    f"{ROOT}/tests/native/exp_bits_check.cpp", "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout == "0\n"
