"""Results are ordinary memory: a copy to a device started out of one is not
changed by what happens to the array afterwards, and blocks are used again
within their bounds."""

import gc

import numpy as np
import pytest


def test_results_are_not_page_locked(monkeypatch):
    from argent_b200 import gpu as G

    monkeypatch.setattr(G.N, "gpu", lambda: pytest.fail("a result asked for page-locked memory"))
    pool = type(G._results)()
    a = pool.array((400, 100, 3), np.float32)
    at, view = a.ctypes.data, a[3:5]
    a[:] = 5.0
    del a
    gc.collect()
    b = pool.array((400, 100, 3), np.float32)
    assert b.ctypes.data != at and (view == 5.0).all()  # a view keeps its block
    del view
    gc.collect()
    c = pool.array((399, 100, 3), np.float32)
    assert c.ctypes.data == at and c.flags.writeable
    pool.IDLE = 1 << 20
    held = [pool.array(1 << 20, np.uint8) for _ in range(3)]
    del held, b, c
    gc.collect()
    assert pool.idle <= pool.IDLE and pool.total == pool.idle == sum(x.size for x in pool._blocks.values())


@pytest.mark.gpu
def test_asynchronous_copies_of_dropped_results():
    """Three hit arrays are sent off with non_blocking while the stream is
    still busy, each dropped at once; the next calls' results must not show in
    the copies."""
    import torch

    from argent_b200 import mesh as M
    from argent_b200.gpu import Context, Piece

    m = M.ring()
    piece = Piece(Context(0), m)
    rng = np.random.default_rng(2)
    rays = np.zeros((1 << 17, 8), np.float32)
    rays[:, :3] = rng.normal(size=(len(rays), 3)) * 30
    rays[:, 3], rays[:, 4:7] = np.inf, -rays[:, :3]
    sets = [np.ascontiguousarray(rays[k * 32768:(k + 1) * 32768]) for k in range(4)]
    want = [piece.trace_closest(r).copy() for r in sets]
    gc.collect()
    torch.zeros(1, device="cuda")
    torch.cuda.synchronize()
    got = []
    for r in sets:
        torch.cuda._sleep(20_000_000)  # about ten milliseconds of other work
        got.append(torch.from_numpy(piece.trace_closest(r)).to("cuda", non_blocking=True))
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        assert np.array_equal(g.cpu().numpy().view(np.uint32), w.view(np.uint32))
    assert not torch.from_numpy(piece.trace_closest(sets[0])).is_pinned()


def test_trim_frees_what_waits():
    from argent_b200 import gpu as G

    pool = type(G._results)()
    held = [pool.array((n, 1 << 18), np.uint8) for n in (1, 2, 3)]
    del held[:2]
    gc.collect()
    assert pool.idle > 0
    pool.trim()
    assert pool.idle == 0 and pool.total == held[0].nbytes and len(pool._blocks) == 1
    held[0][:] = 1


@pytest.mark.gpu
def test_trim_gives_device_scratch_back():
    import torch

    from argent_b200.gpu import Context, denoise_atrous

    ctx = Context(0)
    small = np.ones((8, 8, 3), np.float32)
    want = denoise_atrous(ctx, small)
    ctx.trim()
    free = torch.cuda.mem_get_info(0)[0]
    denoise_atrous(ctx, np.ones((1500, 2000, 3), np.float32))
    assert free - torch.cuda.mem_get_info(0)[0] > 100 << 20  # 28 floats a pixel stay
    ctx.trim()
    assert free - torch.cuda.mem_get_info(0)[0] < 8 << 20
    assert np.array_equal(denoise_atrous(ctx, small), want)
