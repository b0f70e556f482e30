"""The mesh sampler's tree of patches: triangles are cut into leaves of 40, far
points see a patch as its boundary's fan, so meshes of one leaf, of two and more,
split vertices, an open surface and a second, closed component inside the box are
where a wrong boundary would show.  The oracle sums every triangle's solid angle
in FP64; its winding numbers are compared with 1/2 away from rounding (no
candidate point of these meshes lies within 1e-9 of it)."""
import numpy as np
import pytest

import dmpm
from oracle import mesh as omesh

pytestmark = pytest.mark.gpu


def _torus(nu, nv, R=0.5, r=0.21):
    u, v = np.meshgrid(2 * np.pi * np.arange(nu) / nu, 2 * np.pi * np.arange(nv) / nv, indexing="ij")
    P = np.stack([(R + r * np.cos(v)) * np.cos(u), (R + r * np.cos(v)) * np.sin(u), r * np.sin(v)], -1).reshape(-1, 3)
    c, s = np.cos(0.4), np.sin(0.4)
    V = (P @ np.array([[c, -s, 0], [s, c, 0], [0, 0, 1]]) @ np.array([[1, 0, 0], [0, c, s], [0, -s, c]])).astype(np.float32)
    i, j = np.meshgrid(np.arange(nu), np.arange(nv), indexing="ij")
    a, b = i * nv + j, ((i + 1) % nu) * nv + j
    d, e = ((i + 1) % nu) * nv + (j + 1) % nv, i * nv + (j + 1) % nv
    F = np.concatenate([np.stack([a, b, d], -1).reshape(-1, 3), np.stack([a, d, e], -1).reshape(-1, 3)])
    return V, F.astype(np.int32)


def _mesh(kind):
    if kind == "one_leaf":
        return _torus(6, 3)
    if kind == "one_patch":
        return _torus(8, 4)
    if kind == "two_patches":
        return _torus(11, 3)
    V, F = _torus(24, 9)
    if kind == "split_vertices":  # every face with vertices of its own
        return V[F].reshape(-1, 3), np.arange(3 * len(F), dtype=np.int32).reshape(-1, 3)
    if kind == "open":
        return V, F[7:]
    if kind == "two_components":
        W, G = _torus(9, 5, 0.14, 0.05)
        return np.concatenate([V, W]), np.concatenate([F, G + len(V)])
    return V, F


@pytest.mark.parametrize("kind", ["one_leaf", "one_patch", "two_patches", "many", "split_vertices", "open", "two_components"])
def test_sampler_matches_the_sum_over_all_triangles(gpu_ready, kind):
    V, F = _mesh(kind)
    dx = 0.037
    mn, dims, axes = omesh.lattice(V, dx)
    X, Y, Z = np.meshgrid(*axes, indexing="ij")
    P = np.stack([X.ravel(), Y.ravel(), Z.ravel()], axis=1)
    w = omesh.winding_numbers(P, V, F)
    assert np.abs(w - 0.5).min() > 1e-9
    got = dmpm.mesh_lattice_points(V, F, dx)
    assert np.array_equal(got, P[w >= 0.5].astype(np.float32))
