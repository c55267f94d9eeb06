"""A film does not depend on how the planner cut its pass into waves: the film
adds fixed groups of 8 samples, and waves hold whole groups.  Sample counts
around the group and the 32 samples a warp holds, pixel counts that no chunk
divides, waves from a few pixels to the whole pass."""

import numpy as np
import pytest

from argent_b200 import workloads as W


@pytest.mark.gpu
@pytest.mark.parametrize("spp", [1, 7, 8, 9, 31, 33, 40, 100])
def test_film_is_the_same_for_every_wave_size(spp):
    from argent_b200 import _native as N
    from argent_b200.gpu import Context, Film, Piece, Scene, render_pass

    wl = W.ring_still(width=37, height=23)
    want = None
    for wave in (1, 200, 1 << 10, 5000, 0):
        ctx = Context(0, wave_paths=wave, lanes=2)
        piece = Piece(ctx, wl.mesh)
        scene = Scene(ctx, piece, wl.desc)
        films = [Film(ctx, wl.width, wl.height, f) for f in (N.FILM_KAHAN, N.FILM_FP64)]
        got = []
        for f in films:
            render_pass(ctx, scene, wl.camera, f, wl.settings, spp, wl.seed)
            got += [f.xyz(), *f.read()]
        if want is None:
            want = got
        for a, b in zip(got, want):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (wave, spp)
    assert want[0].any() and want[3].any()
