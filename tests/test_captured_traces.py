"""Device-pointer traces captured into graphs: graphs run beside each other and
beside the context's own calls, each with a work counter of its own."""

import ctypes

import numpy as np
import pytest

from tests.rays import make_rays


@pytest.mark.gpu
def test_graphs_of_traces_run_beside_each_other():
    import torch

    from argent_b200 import _native as N
    from argent_b200 import mesh as M
    from argent_b200.gpu import Context, Piece

    m = M.ring()
    ctx = Context(0)
    piece = Piece(ctx, m)
    lib = N.gpu()
    stream = torch.cuda.ExternalStream(ctx.stream)
    sets = [make_rays(m.positions, m.tris, 200_000, seed=40 + k) for k in range(4)]
    want = [(piece.trace_closest(r).view(np.uint32).copy(), piece.trace_anyhit(r).copy()) for r in sets]
    rays = [torch.from_numpy(r).cuda() for r in sets]
    hits = [torch.zeros((len(r), 4), dtype=torch.float32, device="cuda") for r in sets]
    occ = [torch.zeros(len(r), dtype=torch.uint8, device="cuda") for r in sets]
    torch.cuda.synchronize()
    graphs = []
    for r, h, o in zip(rays, hits, occ):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            p = [ctypes.c_void_p(t.data_ptr()) for t in (r, h, o)]
            assert lib.argent_trace_closest_device(ctx.h, piece.h, p[0], len(r), p[1]) == N.OK
            assert lib.argent_trace_anyhit_device(ctx.h, piece.h, p[0], len(r), p[2]) == N.OK
        graphs.append(g)
    streams = [torch.cuda.Stream() for _ in graphs]
    for _ in range(5):
        for t in hits + occ:
            t.zero_()
        torch.cuda.synchronize()
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        assert np.array_equal(piece.trace_closest(sets[1]).view(np.uint32), want[1][0])
        torch.cuda.synchronize()
        for h, o, (wh, wo) in zip(hits, occ, want):
            assert np.array_equal(h.cpu().numpy().view(np.uint32), wh)
            assert np.array_equal(o.cpu().numpy(), wo)
