"""The touch of a caller's pages before a copy into them leaves their bytes as they
are (the copy may still fail) and brings the pages in."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_touch_keeps_the_bytes(tmp_path):
    exe = tmp_path / "touch_check"
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{ROOT}/viennaemc_gb300/csrc",
                    f"{ROOT}/tests/native/touch_check.cpp", "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout == "0 0\n"
    assert "touchRange(dst, bytes);" in (ROOT / "viennaemc_gb300/csrc/emcg_core.cu").read_text()
