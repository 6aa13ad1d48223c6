"""The library is built anew when any of its sources changes."""
import os

from viennaemc_gb300 import _lib


def test_every_source_file_is_watched():
    assert sorted(_lib.SOURCES + _lib.HEADERS) == sorted(
        f for f in os.listdir(_lib.CSRC) if f.endswith((".cu", ".cuh", ".h")))
