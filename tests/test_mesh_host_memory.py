"""The mesh sampler's C entries when host memory runs out (no GPU needed: the
triangles are gathered and cut into patches before the first device call): the
call returns DMPM_ERR_OOM, and no C++ exception ends the process."""
import os
import subprocess
import sys

import pytest

import dmpm

PROG = """
import ctypes, resource, sys
import numpy as np
lib = ctypes.CDLL(sys.argv[1])
nf = 2000000
V = np.random.default_rng(1).random((3000, 3), dtype=np.float32)
F = np.random.default_rng(2).integers(0, 3000, (nf, 3), dtype=np.int32)
mn, mx, n = np.zeros(3, np.float32), np.ones(3, np.float32), ctypes.c_int64()
p = lambda a: ctypes.c_void_p(a.ctypes.data)
held = [int(l.split()[1]) for l in open("/proc/self/status") if l.startswith("VmSize")][0] << 10
resource.setrlimit(resource.RLIMIT_AS, (held + (int(sys.argv[3]) << 20),) * 2)
if sys.argv[2] == "lattice":
    st = lib.dmpm_mesh_lattice_points(p(V), 3000, p(F), nf, p(mn), p(mx), ctypes.c_float(0.01), None,
                                      ctypes.c_int64(0), ctypes.byref(n))
else:
    st = lib.dmpm_mesh_jittered_points(p(V), 3000, p(F), nf, p(mn), p(mx), ctypes.c_float(0.02), 2, ctypes.c_uint64(1),
                                       None, ctypes.c_int64(0), ctypes.byref(n))
print("status", st)
"""


# 2M triangles take 72 MB gathered; their tree a few times that
@pytest.mark.parametrize("call", ["lattice", "jittered"])
@pytest.mark.parametrize("free_mb", [40, 150])
def test_out_of_host_memory_is_an_error_code(call, free_mb):
    dmpm.load_library()
    r = subprocess.run([sys.executable, "-c", PROG, dmpm.LIB_PATH, call, str(free_mb)], capture_output=True, text=True,
                       timeout=300, env=dict(os.environ, OPENBLAS_NUM_THREADS="1"))
    assert r.returncode == 0, r.stderr[-500:]
    assert r.stdout.split() == ["status", str(dmpm.ERR_OOM)]
