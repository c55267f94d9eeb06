"""Ambient occlusion with more samples per vertex than one launch takes (2^30
rays): the samples of a vertex are then split over launches."""

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("samples", [1, 1000, (1 << 30) - 1, 1 << 30, (1 << 30) + 3])
def test_every_sample_of_a_vertex_counts_once(samples):
    """Inside a closed tetrahedron (watertight triangles) every ray is
    occluded: the share is 1 exactly.  Vertices without a normal cast none."""
    from argent_b200 import _native as N
    from argent_b200 import mesh as M
    from argent_b200.gpu import Context, Piece

    pos = np.float32([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]])
    tris = np.uint32([[0, 2, 1], [0, 1, 3], [0, 3, 2], [1, 2, 3]])
    piece = Piece(Context(0), M.Mesh(pos, tris))
    piece.set_triangle_test(N.TRI_WATERTIGHT)
    normals = np.zeros((4, 3), np.float32)
    normals[2] = pos.mean(0) - pos[2]
    assert piece.ambient_occlusion(normals, samples, 5.0).tolist() == [0.0, 0.0, 1.0, 0.0]
