"""Performance cases: the work a user of this library has it do, through the
public Python handles (argent_b200.gpu, argent_b200.workloads).

  listed()            the cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) what a program holds before the call (context, piece,
                      scene, film, host images), made from the seed
  run(state)          one pass, and its whole outputs
  work(case)          bytes and operations one pass cannot do without
  exact(case, seed)   the outputs in 64-bit arithmetic, where they have such
                      a value (the denoiser); None elsewhere

Kinds of case:
  still    film.clear + render_pass + film.read: one render of one piece
           (ring, signet, gem ring, opal ring) in a studio
  reel     render_batch of the alloys of one turntable frame under an
           environment map, rays shared across the alloys or not, films read
  serve    requests submitted to a Serve, stepped until done, all read
  trace    closest hit or any hit of a host array of rays
  ao       ambient occlusion of every vertex of a piece (the patina mask's
           device half)
  denoise  a-trous filter of host images
  develop  tone mapping of a host image to 8 bits
  swap     piece upload with the BVH built on the device, and a sparse grid of
           pick rays traced through it
A context is made once per process and kept, as a program keeps it."""

import math

import numpy as np
import torch

from argent_b200 import _native as N
from argent_b200 import mesh as M
from argent_b200 import workloads as W
from argent_b200 import gpu as G

_CTX = {}


def _context():
    if "ctx" not in _CTX:
        _CTX["ctx"] = G.Context(0)
    return _CTX["ctx"]


def listed():
    return [
        # The autofocus of a shot: eight probe rays through the piece
        # (workloads.shot), the smallest call a program makes.
        {"name": "probes", "kind": "trace", "tris": 500_000, "rays": 8, "any": False},
        # A caller's own rays (visibility and measuring tools): the traversal
        # tests' mixture at 2^20 and a few, on the full-still piece.
        {"name": "rays", "kind": "trace", "tris": 2_097_152, "rays": 1_048_579, "any": False},
        # The small still (ring, 256 x 256, 16 spp, depth 8).
        {"name": "ring_still", "kind": "still", "piece": "ring", "tris": 65_536, "studio": "noir", "width": 256,
         "height": 256, "spp": 16, "depth": 8, "f_stop": 0.0},
        # The served preview on its own: what a look change shows first.
        {"name": "preview", "kind": "still", "piece": "signet", "tris": 500_000, "studio": "noir", "width": 512,
         "height": 512, "spp": 4, "depth": 12, "f_stop": 0.0},
        # The headline still.
        {"name": "signet_still", "kind": "still", "piece": "signet", "tris": 2_097_152, "studio": "noir",
         "width": 1920, "height": 1080, "spp": 256, "depth": 12, "f_stop": 16.0},
        # The gem setting at the gems still's frame and depth, at the sample
        # count of one progressive pass of it.
        {"name": "gems_still", "kind": "still", "piece": "gems", "tris": 928_358, "studio": "white", "width": 1080,
         "height": 1920, "spp": 32, "depth": 32, "f_stop": 0.0},
        # One turntable frame of a reel in four alloys, odd frame size, rays
        # shared across the alloys as a reel renders it.
        {"name": "reel_frame", "kind": "reel", "tris": 1_105_920, "alloys": 4, "share": True, "width": 541,
         "height": 961, "spp": 16, "map": 1024},
        # A burst of requests at the server: previews and one listing.
        {"name": "serve_burst", "kind": "serve", "tris": 250_000, "previews": 8, "size": 512, "spp": 4,
         "listing": 1000, "listing_spp": 16},
        # The patina mask's hemisphere rays at its default 48 per vertex.
        {"name": "patina_ao", "kind": "ao", "tris": 250_000, "samples": 48, "distance": 1.2},
        # A full frame through the denoiser with its guides.
        {"name": "denoise_hd", "kind": "denoise", "width": 1920, "height": 1080, "guides": 2},
        # A listing's frame developed with the default grade.
        {"name": "develop", "kind": "develop", "width": 2000, "height": 2000, "tonemap": "agx", "sat": 1.0},
        # A new piece swapped in while the renderer runs.
        {"name": "piece_swap", "kind": "swap", "tris": 500_000, "probes": 1024},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["still", "still", "still", "reel", "serve", "trace", "ao", "denoise", "develop", "swap"])
    if kind == "still":
        piece = rng.choice(["ring", "signet", "signet", "gems", "opal"])
        w, h = _log(rng, 64, 2000), _log(rng, 64, 2000)
        most = {"ring": 2e8, "signet": 3e8, "gems": 5e7, "opal": 2e7}[piece]
        spp = _log(rng, 1, max(1, min(512, most / (w * h))))
        tris = {"ring": 65_536, "gems": 928_358, "opal": 65_536}.get(piece) or _log(rng, 40_000, 2_097_152)
        return {"kind": "still", "piece": piece, "tris": tris, "studio": rng.choice(["noir", "white"]), "width": w,
                "height": h, "spp": spp, "depth": rng.choice([8, 12, 32]) if piece != "gems" else 32,
                "f_stop": rng.choice([0.0, 16.0])}
    if kind == "reel":
        w, h = _log(rng, 100, 1080), _log(rng, 100, 1920)
        return {"kind": "reel", "tris": _log(rng, 61_440, 1_500_000), "alloys": rng.randint(2, 4),
                "share": rng.random() < 0.7, "width": w, "height": h,
                "spp": _log(rng, 1, max(1, min(64, 4e7 / (w * h)))), "map": rng.choice([512, 1024, 2048])}
    if kind == "serve":
        return {"kind": "serve", "tris": _log(rng, 40_000, 1_000_000), "previews": rng.randint(1, 12),
                "size": _log(rng, 128, 512), "spp": rng.choice([1, 2, 4]), "listing": _log(rng, 300, 2000),
                "listing_spp": rng.choice([4, 8, 16])}
    if kind == "trace":
        return {"kind": "trace", "tris": _log(rng, 40_000, 2_097_152), "rays": _log(rng, 1, 2_000_000),
                "any": rng.random() < 0.5}
    if kind == "ao":
        return {"kind": "ao", "tris": _log(rng, 40_000, 1_000_000), "samples": rng.choice([16, 48, 64]),
                "distance": round(rng.uniform(0.4, 2.5), 3)}
    if kind == "denoise":
        return {"kind": "denoise", "width": _log(rng, 64, 2000), "height": _log(rng, 64, 2000),
                "guides": rng.choice([0, 1, 2, 2])}
    if kind == "develop":
        return {"kind": "develop", "width": _log(rng, 64, 2000), "height": _log(rng, 64, 2000),
                "tonemap": rng.choice(["agx", "aces", "neutral"]), "sat": rng.choice([1.0, 1.15])}
    return {"kind": "swap", "tris": _log(rng, 40_000, 1_000_000), "probes": _log(rng, 64, 4096)}


# ---------------------------------------------------------------- inputs

def _signet(tris, seed):
    """The signet generator at about `tris` triangles (2 * nu * nv, nu about
    three times nv), its emboss and slot mask from the seed."""
    nv = max(8, int(round(math.sqrt(tris / 6.0))))
    nu = max(8, int(round(tris / (2.0 * nv))))
    return M.signet(nu=nu, nv=nv, seed=1 + seed % 1009, mask_seed=2 + seed % 997)


def _still(case, seed, rng, ctx):
    kind, studio = case["piece"], case["studio"]
    w, h = case["width"], case["height"]
    if kind in ("ring", "opal"):
        m = M.ring(seed=1 + seed % 1009)
    elif kind == "gems":
        m = M.gem_ring(seed=4 + seed % 1009)
    else:
        m = _signet(case["tris"], seed)
    piece = G.Piece(ctx, m)
    cam, turn = W.shot(piece, W.hull(m), "hero", 100.0, case["f_stop"], w / h)
    turn += float(rng.uniform(-30.0, 30.0))
    if kind == "gems":
        mats = [W.metal("gold18k", 0.07, 0.8), W.gem("diamond")] + [W.gem(g) for g in W.SIDE_GEMS]
    elif kind == "opal":
        mats = [W.opal(seed % 2 == 1, 0.35)]
    elif kind == "ring":
        mats = [W.metal("sterling", 0.07, 0.8)]
    else:
        mats = [W.metal("gold14k", 0.05, 0.8), W.metal("gold14k", 0.35, 0.8)]
    desc = W._studio_scene(m, mats, studio, turn)
    scene = G.Scene(ctx, piece, desc)
    return {"ctx": ctx, "piece": piece, "scene": scene, "cam": cam, "film": G.Film(ctx, w, h),
            "settings": W.settings(case["depth"]), "spp": case["spp"], "seed": seed & 0x7FFFFFFF}


def _reel(case, seed, rng, ctx):
    w, h = case["width"], case["height"]
    m = _signet(case["tris"], seed)
    piece = G.Piece(ctx, m)
    cam, az = W.turntable_camera(W.hull(m), "hero", 100.0, 0.0, w / h)
    env = W.hdri(case["map"], case["map"] // 2, seed=5 + seed % 1009)
    turn = W.reel_frame_turn(az, int(rng.integers(W.REEL_FRAMES)))
    descs = [W.reel_scene(m, a, env, turn) for a in W.REEL_ALLOYS[: case["alloys"]]]
    scenes = [G.Scene(ctx, piece, d) for d in descs]
    films = [G.Film(ctx, w, h) for _ in scenes]
    ps = W.settings(12)
    items = [(s, cam, f, ps, case["spp"], seed & 0x7FFFFFFF) for s, f in zip(scenes, films)]
    return {"ctx": ctx, "piece": piece, "scenes": scenes, "films": films, "items": items, "share": case["share"]}


def _serve(case, seed, rng, ctx):
    m = _signet(case["tris"], seed)
    piece = G.Piece(ctx, m)
    scenes, reqs = [], []
    cam, turn = W.shot(None, W.hull(m), "hero", 100.0, 0.0, 1.0)
    for i in range(case["previews"] + 1):
        alloy = W.SERVE_ALLOYS[int(rng.integers(len(W.SERVE_ALLOYS)))]
        scenes.append(G.Scene(ctx, piece, W.serve_scene(m, alloy, turn + float(rng.uniform(-40.0, 40.0)))))
        size, spp, pr = ((case["size"], case["spp"], 0) if i < case["previews"]
                         else (case["listing"], case["listing_spp"], 1))
        reqs.append((scenes[-1], cam, W.settings(12), size, size, spp, (seed + i) & 0x7FFFFFFF, pr))
    return {"ctx": ctx, "piece": piece, "scenes": scenes, "reqs": reqs, "serve": G.Serve(ctx, overlap=True)}


def _rays(m, n, rng):
    """Half the rays from a sphere round the piece toward it, half from just
    off its surface into the hemisphere above, some with a finite reach."""
    lo, hi = m.bounds()
    mid, rad = (lo + hi) * 0.5, float(np.linalg.norm(hi - lo)) * 0.5
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    t = mid + rng.uniform(-0.6, 0.6, (n, 3)) * (hi - lo)
    o = t - d * 3.0 * rad
    v = rng.integers(len(m.positions), size=n)
    up = rng.normal(size=(n, 3))
    up /= np.linalg.norm(up, axis=1, keepdims=True)
    up = up * np.where((up * m.normals[v]).sum(1, keepdims=True) < 0, -1.0, 1.0)
    local = (np.arange(n) % 2 == 1)[:, None]
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3] = np.where(local, m.positions[v] + 1e-3 * m.normals[v], o)
    rays[:, 4:7] = np.where(local, up, d)
    rays[:, 3] = np.where(rng.random(n) < 0.25, rng.uniform(0.2, 4.0, n) * rad, np.inf)
    return rays


def _image(w, h, rng):
    """A noisy render's stand-in: albedo in patches, smooth normals, radiance
    with log-normal noise and a few fireflies."""
    y, x = np.mgrid[0:h, 0:w].astype(np.float32)
    k = (np.floor(x / 37.0) * 31 + np.floor(y / 29.0) * 17).astype(np.int64)
    pal = rng.uniform(0.02, 1.0, (257, 3)).astype(np.float32)
    albedo = pal[k % 257]
    fx, fy = rng.uniform(5.0, 40.0, 2)
    n = np.stack([np.sin(x / fx), np.cos(y / fy), np.ones_like(x)], -1)
    normal = (n / np.linalg.norm(n, axis=-1, keepdims=True)).astype(np.float32)
    light = np.exp(0.6 * rng.standard_normal((h, w, 1))) * (0.6 + 0.4 * np.sin(x / (3 * fx) + y / (2 * fy)))[..., None]
    light = np.where(rng.random((h, w, 1)) < 5e-4, light * 200.0, light)
    return (albedo * light).astype(np.float32), albedo, normal


_TONEMAPS = {"agx": 0, "aces": 1, "neutral": 2}


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    ctx = _context()
    if kind in ("still", "reel", "serve"):
        st = {"still": _still, "reel": _reel, "serve": _serve}[kind](case, seed, rng, ctx)
    elif kind == "trace":
        m = _signet(case["tris"], seed)
        st = {"ctx": ctx, "piece": G.Piece(ctx, m), "rays": _rays(m, case["rays"], rng), "any": case["any"]}
    elif kind == "ao":
        m = _signet(case["tris"], seed)
        st = {"ctx": ctx, "piece": G.Piece(ctx, m), "normals": m.normals, "samples": case["samples"],
              "distance": case["distance"]}
    elif kind == "swap":
        m = _signet(case["tris"], seed)
        st = {"ctx": ctx, "mesh": m, "rays": _rays(m, case["probes"], rng)}
    else:
        color, albedo, normal = _image(case["width"], case["height"], rng)
        st = {"ctx": ctx, "color": color}
        if kind == "denoise":
            st["albedo"] = albedo if case["guides"] >= 1 else None
            st["normal"] = normal if case["guides"] >= 2 else None
        else:
            st["grade"] = N.ArgentGrade(0.0, _TONEMAPS[case["tonemap"]], N.AGX_PUNCHY, case["sat"])
    st["kind"] = kind
    return st


def _hits(h):
    return {"tuv": h[:, :3], "prim": h[:, 3].view(np.int32)}


def run(state):
    ctx, kind = state["ctx"], state["kind"]
    if kind == "still":
        film = state["film"]
        film.clear()
        G.render_pass(ctx, state["scene"], state["cam"], film, state["settings"], state["spp"], state["seed"])
        return film.read()
    if kind == "reel":
        for f in state["films"]:
            f.clear()
        ctx.set_ray_sharing(state["share"])
        G.render_batch(ctx, state["items"])
        ctx.set_ray_sharing(False)
        return [f.color() for f in state["films"]]
    if kind == "serve":
        sv = state["serve"]
        tickets = [sv.submit(s, cam, ps, w, h, spp, seed, pr) for s, cam, ps, w, h, spp, seed, pr in state["reqs"]]
        sv.run()
        return [sv.read(t)[0] for t in tickets]
    if kind == "trace":
        if state["any"]:
            return state["piece"].trace_anyhit(state["rays"])
        return _hits(state["piece"].trace_closest(state["rays"]))
    if kind == "ao":
        return state["piece"].ambient_occlusion(state["normals"], state["samples"], state["distance"])
    if kind == "denoise":
        return G.denoise_atrous(ctx, state["color"], state["albedo"], state["normal"])
    if kind == "develop":
        return G.develop(ctx, state["color"], state["grade"])
    piece = G.Piece(ctx, state["mesh"], device_bvh=True)
    lo, hi = piece.bounds()
    hits = piece.trace_closest(state["rays"])
    piece.close()
    return {"lo": lo, "hi": hi, **_hits(hits)}


# ---------------------------------------------------------------- work

# Operations per path-sample that any path tracer of these scenes does:
# about 200 per wide node entered, 60 per triangle, and about 700 per shaded
# bounce (BSDF twice, one light sample), at the counts of rays, nodes and
# bounces the library's own counters give for each piece.
_PATH_FLOPS = {"ring": 2500.0, "signet": 2500.0, "gems": 6000.0, "opal": 5000.0}
_TRI = 36.0  # bytes of three vertices


def work(case):
    kind = case["kind"]
    if kind == "still":
        px = case["width"] * case["height"]
        return {"bytes": px * 36.0 + case["tris"] * _TRI, "flops": px * case["spp"] * _PATH_FLOPS[case["piece"]]}
    if kind == "reel":
        px = case["width"] * case["height"] * case["alloys"]
        k = 1.0 / case["alloys"] if case["share"] else 1.0
        return {"bytes": px * 12.0 + case["tris"] * _TRI + case["map"] ** 2 / 2 * 12.0,
                "flops": px * case["spp"] * 2500.0 * (0.5 + 0.5 * k)}
    if kind == "serve":
        px = case["previews"] * case["size"] ** 2 + case["listing"] ** 2
        ps = case["previews"] * case["size"] ** 2 * case["spp"] + case["listing"] ** 2 * case["listing_spp"]
        return {"bytes": px * 36.0 + case["tris"] * _TRI, "flops": ps * 2500.0}
    if kind == "trace":
        n = case["rays"]
        out = 1.0 if case["any"] else 16.0
        return {"bytes": n * (32.0 + out) + min(case["tris"], 4 * n) * _TRI, "flops": n * 2000.0}
    if kind == "ao":
        nv = case["tris"] / 2
        return {"bytes": nv * 28.0 + case["tris"] * _TRI, "flops": nv * case["samples"] * 800.0}
    px = case["width"] * case["height"] if "width" in case else 0
    if kind == "denoise":
        return {"bytes": px * (24.0 + 12.0 * case["guides"]), "flops": px * 5 * 25 * 30.0}
    if kind == "develop":
        return {"bytes": px * 15.0, "flops": px * 150.0}
    nt = case["tris"]
    return {"bytes": nt * (6.0 + 12.0 + 2.0 + 12.0) + nt * (48.0 + 16.0 + 16.0), "flops": nt * 400.0}


# ---------------------------------------------------------------- 64-bit values

def _blur64(x, taps):
    k = torch.tensor(taps, dtype=torch.float64, device=x.device)
    r = len(taps) // 2
    for d in (1, 0):
        acc, ws = torch.zeros_like(x), torch.zeros_like(x)
        n = x.shape[d]
        for i in range(len(taps)):
            s = i - r
            dst = slice(max(0, -s), min(n, n - s))
            src = slice(max(0, s), min(n, n + s))
            if dst.start >= dst.stop:
                continue
            di, si = [slice(None)] * 2, [slice(None)] * 2
            di[d], si[d] = dst, src
            acc[tuple(di)] += k[i] * x[tuple(si)]
            ws[tuple(di)] += k[i]
        x = acc / ws
    return x


def _lum64(c):
    return c[..., 0] * 0.2126 + c[..., 1] * 0.7152 + c[..., 2] * 0.0722


def exact(case, seed):
    """The denoiser in 64 bits (an edge-avoiding a-trous filter: five passes
    of the 5 x 5 B3 spline, luminance, albedo and normal weights)."""
    if case["kind"] != "denoise":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    color, albedo, normal = _image(case["width"], case["height"], np.random.default_rng(seed))
    t = lambda a: torch.from_numpy(a).to(dev).double()  # noqa: E731
    sig = t(color).clamp(min=0.0)
    a = t(albedo).clamp(0.0, 1.0) if case["guides"] >= 1 else None
    nrm = t(normal) if case["guides"] >= 2 else None
    demod = None
    if a is not None:
        demod = a.clamp(min=float(np.float32(0.02)))
        sig = sig / demod
    if nrm is not None:
        nrm = nrm / nrm.norm(dim=-1, keepdim=True)
    lum = _lum64(sig)
    var = _blur64(1.125 * (lum - _blur64(lum, [1.0] * 3)) ** 2, [1.0] * 5)
    b3 = [1 / 16, 1 / 4, 3 / 8, 1 / 4, 1 / 16]
    h, w = lum.shape
    for p in range(5):
        step = 1 << p
        isl = 1.0 / (4.0 * _blur64(var, [0.25, 0.5, 0.25]).clamp(min=0.0).sqrt() + 1e-10)
        acc, ws, wv = torch.zeros_like(sig), torch.zeros_like(lum), torch.zeros_like(lum)
        for ky in range(5):
            sy = (ky - 2) * step
            dy, qy = slice(max(0, -sy), min(h, h - sy)), slice(max(0, sy), min(h, h + sy))
            if dy.start >= dy.stop:
                continue
            for kx in range(5):
                sx = (kx - 2) * step
                dx, qx = slice(max(0, -sx), min(w, w - sx)), slice(max(0, sx), min(w, w + sx))
                if dx.start >= dx.stop:
                    continue
                D, Q = (dy, dx), (qy, qx)
                e = (lum[Q] - lum[D]).abs() * isl[D]
                if a is not None:
                    e = e + ((a[D] - a[Q]) ** 2).sum(-1) * 100.0
                g = b3[ky] * b3[kx] * torch.exp(-e)
                if nrm is not None:
                    g = g * (nrm[D] * nrm[Q]).sum(-1).clamp(min=0.0) ** 128
                acc[D] += g[..., None] * sig[Q]
                ws[D] += g
                wv[D] += g * g * var[Q]
        sig, var = acc / ws[..., None], wv / (ws * ws)
        lum = _lum64(sig)
    return (sig * demod if demod is not None else sig).cpu()
