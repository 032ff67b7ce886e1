"""Circuit compilation where the host can start no further threads."""
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]

CODE = """
import ctypes as C, resource, sys
sys.path[:0] = [{pkg!r}]
import numpy as np
from strata_b200 import _lib as L
from strata_b200.gpu import CircuitParts, ProofSets
lib = L.load()
ps = ProofSets.from_lists([[[1, 2], [2, 3]]] * 64)
out = C.c_void_p()
u64, i64 = C.POINTER(C.c_uint64), C.POINTER(C.c_int64)
size = next(int(x.split()[1]) for x in open("/proc/self/status") if x.startswith("VmSize")) << 10
resource.setrlimit(resource.RLIMIT_STACK, (64 << 20, resource.RLIM_INFINITY))  # each thread's stack
resource.setrlimit(resource.RLIMIT_AS, (size + (48 << 20), resource.RLIM_INFINITY))
rc = lib.strata_circuits_compile_host(len(ps), ps.proof_off.ctypes.data_as(u64), ps.lit_off.ctypes.data_as(u64),
                                      ps.lits.ctypes.data_as(i64), 4, 0, C.byref(out))
assert rc == 0, rc
parts = CircuitParts(lib, out, len(ps))
assert np.array_equal(parts.eval64(np.full(4, 0.5)), np.full(64, 0.375))
"""


def test_compile_without_threads():
    # 48 MB of address space left, 64 MB for a thread's stack
    r = subprocess.run([sys.executable, "-c", CODE.format(pkg=str(ROOT / "strata-k_b200"))], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stderr[-400:])
