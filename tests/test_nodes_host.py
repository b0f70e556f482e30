"""Node addresses of the FP32 gathers (csrc/kernels_chunk.cuh: StencilNodes),
compiled for the host: dmpm_set_grid takes grids of up to 2e9 nodes, so the record
index of a stencil row (two records of 16 bytes per node in the adjoint gather)
passes 2^31, and so does the span of one stencil on a grid of few, large planes."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "a-differentiable-material-point-method-for-shape-morphing_b200", "csrc")
SRC = os.path.join(HERE, "native", "nodes_host.cu")
LIB = os.path.join(HERE, "native", "libnodes_host.so")


@pytest.fixture(scope="module")
def nh():
    deps = [SRC] + [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    if not os.path.exists(LIB) or any(os.path.getmtime(d) > os.path.getmtime(LIB) for d in deps):
        subprocess.check_call(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17",
                               "-Xcompiler", "-fPIC", "-shared", "-I", CSRC, "-o", LIB, SRC])
    lib = ctypes.CDLL(LIB)
    lib.nh_record.restype = ctypes.c_longlong
    lib.nh_record.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p] + [ctypes.c_int] * 4
    return lib


@pytest.mark.parametrize("dims", [(3, 5, 7), (2, 23000, 23000), (1, 40000, 40000), (2, 31000, 31000), (5, 20000, 20000),
                                  (1240, 1240, 1240)])
def test_rows_of_nodes_inside_the_grid(nh, dims):
    d = np.array(dims, dtype=np.int32)
    goff = 0 if np.prod(d.astype(np.int64)) > 10 ** 6 else 2 ** 31 - 200  # a batch's grids together: below 2^31 nodes
    axes = [sorted({-4, -3, -2, -1, 0, int(n) // 2, int(n) - 4, int(n) - 3, int(n) - 1}) for n in dims]
    seen = 0
    for b0 in axes[0]:
        for b1 in axes[1]:
            for b2 in (-3, 0, dims[2] - 4, dims[2] - 1):
                base = np.array([b0, b1, b2], dtype=np.int32)
                for i in range(4):
                    for j in range(4):
                        gi, gj = b0 + i, b1 + j
                        if not (0 <= gi < dims[0] and 0 <= gj < dims[1]):
                            continue  # no node of this row is read
                        node = (gi * dims[1] + gj) * dims[2] + b2 + goff
                        for pair in (0, 1):
                            whole = all(0 <= b and b + 3 < n for b, n in zip((b0, b1, b2), dims))
                            for inside in (0, 1) if whole else (0,):
                                got = nh.nh_record(d.ctypes.data, goff, base.ctypes.data, i, j, pair, inside)
                                assert got == node * (1 + pair), (dims, base, i, j, pair)
                                seen += 1
    assert seen > 100  # rows were compared
