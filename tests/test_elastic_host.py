"""The closed form of the reference-style stress derivative that the FP32 path's finalize
takes (d2_mult_from_polar<false, false>), compiled for the host, against the same
derivative in extended precision: d(J F^-T) as the derivative of F's cofactors, which the
reference approximates by central differences (Elasticity.cpp:126-140), and dR from
(tr(S) I - S) x = axial(R^T dF - dF^T R).  The form with the differences
(d2_mult_from_polar<false, true>, the FP64 path) is held to the same values where det F is
not small: its quotients divide the rounding of J F^-T, which grows with 1 / det F, by 2e-6."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "a-differentiable-material-point-method-for-shape-morphing_b200", "csrc")
SRC = os.path.join(HERE, "native", "elastic_host.cu")
LIB = os.path.join(HERE, "native", "libelastic_host.so")
LAM, MU = 58.0, 39.0
EPS = 2.3e-16
Q = np.longdouble


@pytest.fixture(scope="module")
def eh():
    deps = [SRC] + [os.path.join(CSRC, f) for f in ("mat3.cuh", "svd3.cuh", "elasticity.cuh")]
    if not os.path.exists(LIB) or any(os.path.getmtime(d) > os.path.getmtime(LIB) for d in deps):
        subprocess.check_call(["/usr/local/cuda/bin/nvcc", "-O2", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                               "-Wno-deprecated-gpu-targets", "-I", CSRC, "-o", LIB, SRC])
    lib = ctypes.CDLL(LIB)
    P = ctypes.c_void_p
    lib.eh_d2.argtypes = [P, P, P, ctypes.c_double, ctypes.c_double, P, ctypes.c_int, P]
    return lib


def _rot(rng):
    q, r = np.linalg.qr(rng.normal(size=(3, 3)))
    q = q * np.sign(np.diag(r))
    return q if np.linalg.det(q) > 0 else q[:, [1, 0, 2]]


def _cof(F, D=None):
    """cofactors of F, or their derivative in the direction D"""
    C = np.zeros((3, 3), Q)
    for i in range(3):
        for j in range(3):
            a, b, c, d = (i + 1) % 3, (i + 2) % 3, (j + 1) % 3, (j + 2) % 3
            if D is None:
                C[i, j] = F[a, c] * F[b, d] - F[a, d] * F[b, c]
            else:
                C[i, j] = D[a, c] * F[b, d] + F[a, c] * D[b, d] - D[a, d] * F[b, c] - F[a, d] * D[b, c]
    return C


def _exact(F, R, S, dF):
    F, R, S, D = (a.astype(Q) for a in (F, R, S, dF))
    C = _cof(F)
    det = (C * F).sum() / 3
    J = max(det, Q(1e-6))
    W = R.T @ D - D.T @ R
    A = np.trace(S) * np.eye(3) - S
    Ac = _cof(A)
    x = Ac.T @ np.array([W[2, 1], W[0, 2], W[1, 0]]) / ((Ac * A).sum() / 3)
    X = np.array([[0, -x[2], x[1]], [x[2], 0, -x[0]], [-x[1], x[0], 0]])
    return 2 * MU * D + LAM * (J / det) ** 2 * (C * D).sum() * C + LAM * (J - 1) * _cof(F, D) - 2 * MU * R @ X


# singular values; the last of a negative determinant carries the sign, as the polar factors do
@pytest.mark.parametrize("s", [(1.0, 1.0, 1.0), (1.01, 1.0, 0.98), (2.0, 1.1, 0.4), (1.5, 0.9, 1e-3), (1.0, 0.9, 1e-5),
                               (1.0, 0.8, 5e-7), (0.02, 0.01, 4e-3), (1.2, 1.0, -0.3), (30.0, 20.0, 10.0)])
def test_closed_form(eh, s):
    rng = np.random.default_rng(int(1e6 * abs(s[2])) + 3)
    det, f = np.prod(s), max(abs(v) for v in s)
    J, cof = max(det, 1e-6), max(abs(s[0] * s[1]), abs(s[0] * s[2]), abs(s[1] * s[2]))
    pairs = [abs(p) for p in (s[0] + s[1], s[0] + s[2], s[1] + s[2])]
    cond = max(pairs) / min(pairs)
    for _ in range(200):
        U, V = _rot(rng), _rot(rng)
        F = np.ascontiguousarray(U @ np.diag(s) @ V.T)
        R, S = np.ascontiguousarray(U @ V.T), np.ascontiguousarray(V @ np.diag(s) @ V.T)
        dF = rng.normal(size=(3, 3))
        d = np.abs(dF).max()
        want = _exact(F, R, S, dF)
        got = np.zeros((3, 3))
        eh.eh_d2(F.ctypes.data, R.ctypes.data, S.ctypes.data, LAM, MU, dF.ctypes.data, 0, got.ctypes.data)
        # products of two entries to a few eps f^2, sums of nine; the clamped quotient (J / det)^2 has
        # det to eps f^3 / det; the system's solution to eps cond^2
        clamp = (J / det) ** 2 * (1 + (6 * f ** 3 / abs(det) if det <= 1e-6 else 0))
        tol = 60 * EPS * d * (LAM * 9 * f * f * f * f * clamp + LAM * (abs(J - 1) + f ** 3) * 9 * f + 2 * MU * cond ** 2 * f / min(f, 1.0))
        assert np.abs(got - want).max() <= tol
        if det > 0.1 or det < -0.1:
            eh.eh_d2(F.ctypes.data, R.ctypes.data, S.ctypes.data, LAM, MU, dF.ctypes.data, 1, got.ctypes.data)
            # an entry of J F^-T to eps (f^2 + f^2 f^3 / det), twice, over 2e-6, nine times
            noise = 9 * d * 2 * 10 * EPS * f * f * (1 + f ** 3 / abs(det)) / 2e-6
            assert np.abs(got - want).max() <= tol + LAM * abs(J - 1) * noise
