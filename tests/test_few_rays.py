"""Small traces and short queues are traversed by eight lanes per ray
(coop_trace): calls of up to four rays per resident warp.  Their hits are
those of the one-thread-per-ray form bit for bit, which larger calls take."""

import numpy as np
import pytest

from tests.rays import make_rays


def _limit(ctx):
    """Rays at which the one-thread-per-ray form starts: 4 per warp, 4 warps
    per block, 8 blocks per SM."""
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count * 8 * 4 * 4


@pytest.mark.gpu
@pytest.mark.parametrize("test", ["moller_trumbore", "watertight"])
@pytest.mark.parametrize("mesh", ["ring", "one", "five"])
def test_few_rays_equal_many(mesh, test):
    """1, 8, 9, one per warp and around it, the most the form takes and one
    more (already the other form), against the same rays inside a call of
    2^16: t, u, v and the triangle, and occlusion, are equal bit for bit."""
    from argent_b200 import _native as N
    from argent_b200 import mesh as M
    from argent_b200.gpu import Context, Piece

    m = M.ring()
    if mesh != "ring":
        k = 1 if mesh == "one" else 5
        m = M.Mesh(m.positions, m.tris[:k], m.normals, m.tri_material[:k])
    ctx = Context(0)
    piece = Piece(ctx, m)
    piece.set_triangle_test(N.TRI_WATERTIGHT if test == "watertight" else N.TRI_MOLLER_TRUMBORE)
    rays = make_rays(m.positions, m.tris, 1 << 16, seed=31)
    rays[::5, 3] = 7.5  # finite reach
    hits, occ = piece.trace_closest(rays), piece.trace_anyhit(rays)
    lim = _limit(ctx)
    assert lim < len(rays)
    for n in (1, 8, 9, lim // 4 - 1, lim // 4 + 1, lim // 2 + 3, lim, lim + 1):
        sub = np.ascontiguousarray(rays[-n:])
        assert np.array_equal(piece.trace_closest(sub).view(np.uint32), hits[-n:].view(np.uint32)), n
        assert np.array_equal(piece.trace_anyhit(sub), occ[-n:]), n
    assert (hits[:, 3].view(np.uint32) != 0xFFFFFFFF).any()
