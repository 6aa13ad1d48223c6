"""emcg_poisson_solve_noalloc from a thread with little stack: the host side keeps its
copy of the boundaries and the levels' descriptors there, under 64 KB in all.  In a
process of its own, which an overflow ends.  Without a GPU the call goes as far as the
device's address and returns its CUDA error; with one, in each form of the solve (one
cluster, a cluster below finer levels, one launch per phase)."""
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CALL = """
import ctypes as C, sys, threading
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
from viennaemc_gb300 import _lib as L
from test_gpu_poisson_large import _bar, _start
lib, out = L.lib(), []
calls = []
for nx, ny, gates in {grids}:
    dev = _bar(nx, ny, gates)
    pot, conc = _start(dev, nx)
    if {gpu}:
        import torch
        d_pot, d_conc = (torch.tensor(v, device="cuda") for v in (pot, conc))
        torch.cuda.synchronize()
        at = d_pot.data_ptr(), d_conc.data_ptr()
    else:
        d_pot = d_conc = None
        at = pot.ctypes.data, conc.ctypes.data  # (never followed)
    calls.append((dev, dev.desc(), d_pot, d_conc, at))

def solve():
    rel, cyc = C.c_double(), C.c_int32()
    for _, desc, _, _, at in calls:
        out.append(lib.emcg_poisson_solve_noalloc(
            C.byref(desc), C.c_void_p(at[0]), C.c_void_p(at[1]), 1, 0, 1e-8, 200, None,
            C.byref(rel), C.byref(cyc)))

solve()  # the runtime's own first-use work, on the main thread
threading.stack_size({stack})
t = threading.Thread(target=solve)
t.start()
t.join()
print(*out)
"""


def _run(gpu, stack, grids):
    code = CALL.format(root=str(ROOT), gpu=gpu, stack=stack, grids=grids)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    return r.returncode, r.stdout.split(), r.stderr


def test_call_without_a_gpu():
    import torch
    if torch.cuda.is_available():
        pytest.skip("the host arrays stand for device memory")
    assert _run(False, 128 << 10, [(201, 101, 0)])[:2] == (0, ["-2", "-2"])


@pytest.mark.gpu
def test_solves_on_a_small_stack(engine):
    rc, out, err = _run(True, 192 << 10, [(201, 101, 0), (360, 361, 0), (301, 61, 61)])
    assert (rc, out) == (0, ["0"] * 6), err
