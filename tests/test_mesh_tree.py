"""The mesh sampler on either side of the candidate count from which it builds its
tree of patches (100,000): below, the triangles are summed as one leaf; from there
on, by the tree's fans and leaves.  Meshes of one leaf, of two and more, split
vertices, an open surface and a second component, on a lattice of either size.  The
oracle sums every triangle's solid angle in FP64 at a random part of the candidates;
winding numbers within 1e-9 of 1/2 are left out."""
import numpy as np
import pytest

import dmpm
from oracle import mesh as omesh
from tests.test_mesh_patches import _mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dx,tree", [(0.0213, True), (0.0265, False)])
@pytest.mark.parametrize("kind", ["one_leaf", "one_patch", "two_patches", "many", "split_vertices", "open", "two_components"])
def test_kept_candidates(gpu_ready, kind, dx, tree):
    V, F = _mesh(kind)
    mn, dims, axes = omesh.lattice(V, dx)
    total = int(np.prod(dims))
    assert (total >= 100000) == tree
    X, Y, Z = np.meshgrid(*axes, indexing="ij")
    P = np.stack([X.ravel(), Y.ravel(), Z.ravel()], axis=1)
    got = dmpm.mesh_lattice_points(V, F, dx)
    at = {p.tobytes(): i for i, p in enumerate(P.astype(np.float32))}
    kept = np.array([at[p.tobytes()] for p in got])  # every point is a candidate
    assert np.all(np.diff(kept) > 0)  # in lattice order
    mask = np.zeros(total, dtype=bool)
    mask[kept] = True
    q = np.random.default_rng(11).choice(total, 6000, replace=False)
    w = omesh.winding_numbers(P[q], V, F)
    clear = np.abs(w - 0.5) > 1e-9
    assert clear.sum() > 5900
    assert np.array_equal(mask[q][clear], (w >= 0.5)[clear])
