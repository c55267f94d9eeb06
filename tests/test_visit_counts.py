"""The traversal's counters mean the same in the form for few rays (eight lanes
per ray) as in the general one: every node visit is in the histogram of
children entered, and the closest hits of the same rays, which visit the same
nodes in the same order, count the same in both."""

import numpy as np
import pytest

from tests.rays import make_rays


@pytest.mark.gpu
@pytest.mark.parametrize("mesh", ["ring", "five"])
def test_both_forms_count_alike(mesh):
    from argent_b200 import mesh as M
    from argent_b200.gpu import Context, Piece

    m = M.ring()
    if mesh == "five":
        m = M.Mesh(m.positions, m.tris[:5], m.normals, m.tri_material[:5])
    ctx = Context(0)
    piece = Piece(ctx, m)
    rays = make_rays(m.positions, m.tris, 1 << 16, seed=19)  # above the few-rays limit as one call
    few = [np.ascontiguousarray(rays[k:k + 8192]) for k in range(0, len(rays), 8192)]
    counts = []
    for calls in ([rays], few):
        ctx.set_counting(True)
        for r in calls:
            piece.trace_closest(r)
            piece.trace_anyhit(r)
        n, h, v = ctx.traversal_counts(), ctx.child_hit_histogram(), ctx.traversal_histogram()
        ctx.set_counting(False)
        assert n["closest_rays"] == n["any_rays"] == len(rays)
        assert sum(h["closest"]) == n["closest_nodes"] > 0 and sum(h["any"]) == n["any_nodes"] > 0
        assert sum(v["closest"]) == sum(v["any"]) == len(rays)
        assert n["any_tris"] > 0
        counts.append((n, h, v))
    (n0, h0, v0), (n1, h1, v1) = counts
    for k in ("closest_rays", "closest_nodes", "closest_tris"):
        assert n0[k] == n1[k], k
    assert h0["closest"] == h1["closest"] and v0["closest"] == v1["closest"]
    if mesh == "five":  # two leaves under one node: the order of visits is the same for any hits too
        assert n0["any_nodes"] == n1["any_nodes"]
