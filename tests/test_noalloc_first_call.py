"""One emcg_poisson_solve_noalloc call at start-up takes all the device memory that
later calls need, whatever form of the solve their grids take (kernels are loaded at
their first use).  In a process of its own, where no other solve has run."""
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CALL = """
import ctypes as C, sys
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
import torch
from viennaemc_gb300 import _lib as L
from test_gpu_poisson_large import _bar, _start
lib, taken, sets = L.lib(), [], []
for nx, ny, gates in {grids}:
    dev = _bar(nx, ny, gates)
    pot, conc = (torch.tensor(v, device="cuda") for v in _start(dev, nx))
    sets.append((dev.desc(), pot, conc, dev))
torch.cuda.synchronize()
for desc, pot, conc, dev in sets:
    before = torch.cuda.mem_get_info()[0]
    rel, cyc = C.c_double(), C.c_int32()
    L.check(lib.emcg_poisson_solve_noalloc(
        C.byref(desc), C.c_void_p(pot.data_ptr()), C.c_void_p(conc.data_ptr()), 1, 0, 1e-8,
        200, None, C.byref(rel), C.byref(cyc)))
    taken.append(before - torch.cuda.mem_get_info()[0])
print(*taken)
"""


@pytest.mark.gpu
def test_first_call_takes_all_memory(engine):
    # one cluster, with held and with column sweeps; a tail; one launch per phase
    grids = [(201, 101, 0), (401, 201, 0), (360, 361, 0), (301, 61, 61), (201, 101, 0)]
    r = subprocess.run([sys.executable, "-c", CALL.format(root=str(ROOT), grids=grids)],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    taken = [int(v) for v in r.stdout.split()]
    assert taken[0] > 0 and taken[1:] == [0, 0, 0, 0]
