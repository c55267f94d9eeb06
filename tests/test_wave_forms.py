"""How a batch is launched by its number of waves: one or two fork the shading
classes and the shadow rays, three and four the shadow rays, more run each lane
in order and are captured as a graph.  Contexts get small waves, so that small
renders take each form, and graph counts show that a graph was captured and
replayed where one should be."""

import numpy as np
import pytest

from argent_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _gem_desc(m):
    mats = [W.metal("gold18k", 0.07, 0.8), W.gem("diamond")] + [W.gem(g) for g in W.SIDE_GEMS]
    return W._studio_scene(m, mats, "white", 20.0)


@pytest.mark.parametrize("kind", ["ring", "gems", "reel"])
def test_films_are_the_same_in_every_form(kind):
    """One to six waves of one pass: the same film bit for bit, the number of
    waves read off the launches, and a graph from five waves on."""
    from argent_b200 import mesh as M
    from argent_b200.gpu import Context, Film, Piece, Scene, render_pass

    w, h, spp = 64, 60, 32
    if kind == "ring":
        wl = W.ring_still(width=w, height=h)
        m, desc, cam = wl.mesh, wl.desc, wl.camera
    else:
        m = M.gem_ring() if kind == "gems" else W.reel_piece("61k")
        desc = _gem_desc(m) if kind == "gems" else W.reel_scene(m, "bronze", W.hdri(256, 128), 30.0)
        cam, _ = W.turntable_camera(W.hull(m), aspect=w / h)
    ps = W.settings(8)
    want, per_wave = None, None
    for waves in (1, 2, 3, 4, 5, 6):
        # 3840 pixels divide by 1 to 6, and each wave takes whole pixels.
        ctx = Context(0, wave_paths=w * h * spp // waves, lanes=4)
        piece = Piece(ctx, m)
        scene = Scene(ctx, piece, desc)
        for repeat in range(2):
            n0 = ctx.kernel_launches
            film = Film(ctx, w, h)
            render_pass(ctx, scene, cam, film, ps, spp, 7)
            got = [film.xyz(), *film.read()]
            launches = ctx.kernel_launches - n0
            if want is None:
                want = got
                per_wave = launches
            for a, b in zip(got, want):
                assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (waves, repeat)
        # A read adds its own few launches; a wave's are far more.
        assert round(launches / per_wave) == waves, (launches, per_wave)
        assert ctx.graph_counts() == ((1, 2) if waves > 4 else (0, 0)), waves


def test_a_captured_graph_is_replayed():
    """New films and another seed replay one graph; without graphs the films
    are the same."""
    from argent_b200.gpu import Context, Film, Piece, Scene, render_pass

    wl = W.ring_still()
    ctx = Context(0, wave_paths=1 << 16)
    piece = Piece(ctx, wl.mesh)
    scene = Scene(ctx, piece, wl.desc)

    def film(seed):
        f = Film(ctx, wl.width, wl.height)
        render_pass(ctx, scene, wl.camera, f, wl.settings, 8, seed)
        return f.xyz()

    ctx.set_graphs(False)
    want = [film(wl.seed), film(wl.seed + 1)]
    assert ctx.graph_counts() == (0, 0) and not np.array_equal(*want)
    ctx.set_graphs(True)
    for k in range(4):
        assert np.array_equal(film(wl.seed + k % 2), want[k % 2])
        assert ctx.graph_counts() == (1, k + 1)


def test_graphs_of_map_and_gradient_waves():
    """Waves of two renders whose scenes do not trace alike (another turntable
    angle), so that a wave names no single scene: gradient-studio scenes first,
    then env-map scenes of the same piece, materials and sizes.  The second
    batch captures a graph of its own."""
    from argent_b200.gpu import Context, Film, Piece, Scene, render_batch

    m = W.reel_piece("61k")
    env = W.hdri(256, 128)
    radius, floor_y = W.piece_radius(m)
    cam, _ = W.turntable_camera(W.hull(m), aspect=1.0)
    ps = W.settings(8)

    def desc(with_map, turn):
        if with_map:
            return W.reel_scene(m, "bronze", env, turn)
        panels, grad, fm, fl, white = W.studio("noir", radius, floor_y)
        mats = [W.metal("bronze", 0.05, 0.8), W.metal("bronze", 0.35, 0.8), fm]
        fl.material = len(mats) - 1
        return W.SceneDesc(mats, panels, grad, fl, turn, white)

    size, spp = 64, 8
    ctx = Context(0, wave_paths=2 * size * size * spp)
    piece = Piece(ctx, m)
    batches = [[Scene(ctx, piece, desc(with_map, turn)) for turn in (30.0, 55.0)] for with_map in (False, True)]

    def render(scenes):
        films = [Film(ctx, size, size) for _ in range(10)]  # five waves of both scenes
        render_batch(ctx, [(scenes[k % 2], cam, f, ps, spp, 7 + k) for k, f in enumerate(films)])
        return [f.xyz() for f in films]

    ctx.set_graphs(False)
    want = [render(b) for b in batches]
    assert not np.array_equal(want[0][0], want[1][0])
    ctx.set_graphs(True)
    for repeat in range(2):
        for k, (b, w) in enumerate(zip(batches, want)):
            for got, ref in zip(render(b), w):
                assert np.array_equal(got, ref)
            assert ctx.graph_counts() == ((k + 1, k + 1) if repeat == 0 else (2, k + 3))


@pytest.mark.parametrize("away", [1.0, 1e3, 1e5])
def test_camera_rays_of_a_far_camera(away):
    """A small render's camera rays take eight lanes each, in a wave with a
    larger render a lane each: the same hits, so the same film, also from so far
    that hits and boxes are off by more than the panels and the floor are apart
    (the camera moved back with its picture kept)."""
    from argent_b200 import mesh as M
    from argent_b200.gpu import Context, Film, Piece, Scene, render_batch, render_pass

    m = M.ring()
    ctx = Context(0)
    piece = Piece(ctx, m)
    cam, turn = W.shot(piece, W.hull(m), "hero", 100.0, 0.0, 1.0)
    scene = Scene(ctx, piece, W._studio_scene(m, [W.metal("sterling", 0.07, 0.8)], "white", turn + 13.0))
    dist = -float(np.dot(cam.pos, cam.forward))
    for i in range(3):
        cam.pos[i] -= cam.forward[i] * dist * (away - 1.0)
    cam.half_w /= away
    cam.half_h /= away
    ps = W.settings(3)
    for seed in range(24):  # 7744 camera rays: four per resident warp at most
        alone, among, other = Film(ctx, 44, 44), Film(ctx, 44, 44), Film(ctx, 256, 256)
        render_pass(ctx, scene, cam, alone, ps, 4, seed)
        render_batch(ctx, [(scene, cam, among, ps, 4, seed), (scene, cam, other, ps, 4, seed)])
        for a, b in zip([alone.xyz(), *alone.read()], [among.xyz(), *among.read()]):
            assert a.any() and np.array_equal(a.view(np.uint32), b.view(np.uint32))
