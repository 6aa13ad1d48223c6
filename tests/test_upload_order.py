"""The engines' streams do not wait for the null stream, and a cudaMemcpy from
pageable memory returns before its transfer: so what an engine uploads, and the
memory it clears, goes through its own stream.  (The host-array Coulomb sums run on
the null stream themselves.)"""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "viennaemc_gb300" / "csrc"


@pytest.mark.parametrize("path", sorted(p.name for p in CSRC.iterdir()
                                        if p.suffix in (".cu", ".cuh", ".h")
                                        and p.name != "emcg_p2p.cu"))
def test_no_upload_or_clear_on_the_null_stream(path):
    code = re.sub(r"//[^\n]*", "", (CSRC / path).read_text())
    assert not re.findall(r"\bcudaMemset\s*\(", code)
    for args in re.findall(r"\bcudaMemcpy\s*\(([^;]*);", code):
        assert "HostToDevice" not in args, args
    # an asynchronous upload or clear names its stream
    for call, args in re.findall(r"\b(cudaMemcpyAsync|cudaMemsetAsync)\s*\(([^;]*);", code):
        depth, commas = 0, 0
        for c in args:
            depth += (c in "([{") - (c in ")]}")
            if depth < 0:
                break
            commas += c == "," and depth == 0
        assert commas == (4 if call == "cudaMemcpyAsync" else 3), (call, args)
