"""The arithmetic that decides which boxes a ray enters is fixed: correctly
rounded inverses, plane bytes decoded exactly, one rounding per plane, an
interval widened by 2^-18 of its magnitude.  A triangle seen edge-on can pass
the triangle test at a point outside its own box, so which of such hits are
found depends on the boxes a ray enters, and any other rounding of the planes
moves some of them (about one camera ray in 10^9 of a still)."""

import hashlib
from fractions import Fraction

import numpy as np
import pytest

from tests import device_host

f = np.float32

PROGRAM = r"""
#include <cstdio>
#include "argent_b200/csrc/device/traverse.cuh"
// Input: a count, then per case a ray (o, d), a reach and a node (20 words).
// Output per case: the three inverses, then for each child whether it is
// entered and its entry distance.
int main() {
  uint32_t n;
  if (fread(&n, 4, 1, stdin) != 1) return 1;
  for (uint32_t i = 0; i < n; ++i) {
    float ray[7];
    uint4 node[5];
    if (fread(ray, 4, 7, stdin) != 7 || fread(node, 16, 5, stdin) != 5) return 1;
    const dev::RayQ r = dev::make_rayq(dev::V3{ray[0], ray[1], ray[2]}, dev::V3{ray[3], ray[4], ray[5]});
    const dev::NodeQ q = dev::node_ray(dev::load_node(node, 0), r);
    float out[19] = {r.ix, r.iy, r.iz};
    for (int c = 0; c < 8; ++c) out[11 + c] = dev::child_q(q, c, ray[6], &out[3 + c]) ? 1.0f : 0.0f;
    fwrite(out, 4, 19, stdout);
  }
}
"""


def _round(x):
    """A rational rounded to float32 (nearest, ties to even) in the range the
    cases use, where nothing overflows or is subnormal."""
    if x == 0:
        return f(0)
    s, x = (-1, -x) if x < 0 else (1, x)
    e = x.numerator.bit_length() - x.denominator.bit_length()
    if Fraction(2) ** e > x:
        e -= 1
    m = x / Fraction(2) ** (e - 23)
    k = m.numerator // m.denominator
    rest = m - k
    if rest > Fraction(1, 2) or (rest == Fraction(1, 2) and k % 2):
        k += 1
    return f(s * float(Fraction(k) * Fraction(2) ** (e - 23)))


def _child(ray, node, inv, c):
    """Entry distance and whether child c is entered, by the rule."""
    lo, hi = [f(0)], [ray[6]]
    for a in range(3):
        origin = node[:3].view(f)[a]
        scale = f(2.0) ** f(int(node[3] >> (8 * a) & 0xFF) - 127)
        ql, qh = (int(node[8 + 2 * k + c // 4] >> (8 * (c % 4)) & 0xFF) for k in (a, 3 + a))
        dd = origin - ray[a]
        b, e = dd * inv[a], ((abs(dd) + f(256) * scale) * abs(inv[a])) * f(2.0**-18)
        k = scale * inv[a]
        near, far = (qh, ql) if np.signbit(inv[a]) else (ql, qh)
        lo.append(_round(Fraction(near) * Fraction(float(k)) + Fraction(float(b - e))))
        hi.append(_round(Fraction(far) * Fraction(float(k)) + Fraction(float(b + e))))
    return max(lo), max(lo) <= min(hi)


def test_planes_and_inverses_are_rounded_once(tmp_path):
    rng = np.random.default_rng(7)
    n = 700
    rays = np.zeros((n, 7), f)
    d = rng.normal(size=(n, 3))
    d[::7, 0] *= 2.0 ** -rng.integers(1, 60, size=len(d[::7]))
    d[3::50, 1] = 0.0
    rays[:, 3:6] = d / np.sqrt((d * d).sum(1, keepdims=True))
    nodes = np.zeros((n, 20), np.uint32)
    size = 2.0 ** rng.uniform(-14, 6, (n, 1))
    nodes[:, :3] = (rng.normal(size=(n, 3)) * 20).astype(f).view(np.uint32)
    ex = np.clip(np.floor(np.log2(size)).astype(int) + rng.integers(-9, -6, (n, 3)), -60, 30) + 127
    nodes[:, 3] = ex[:, 0] | ex[:, 1] << 8 | ex[:, 2] << 16
    q = np.sort(rng.integers(0, 256, (2, n, 3, 8)), axis=0)
    for s in range(2):
        for a in range(3):
            for h in range(2):
                nodes[:, 8 + 6 * s + 2 * a + h] = sum(q[s, :, a, 4 * h + i].astype(np.uint32) << 8 * i
                                                      for i in range(4))
    # Toward the box, so that children are entered and passed closely.
    scale = 2.0 ** (ex - 127.0)
    at = nodes[:, :3].view(f) + scale * rng.uniform(0, 255, (n, 3))
    rays[:, :3] = at - rays[:, 3:6] * size * rng.uniform(0.5, 200, (n, 1))
    rays[:, 6] = np.where(rng.random(n) < 0.5, np.inf, size[:, 0] * 100)
    exe = device_host.compile_program(PROGRAM, tmp_path)
    data = np.uint32(n).tobytes() + np.hstack([rays.view(np.uint32), nodes]).tobytes()
    got = np.frombuffer(device_host.run(exe, data), f).reshape(n, 19)
    cap = f(2.0**64)
    entered = 0
    for i in range(n):
        inv = [cap * (-1 if np.signbit(x) else 1) if abs(x) < f(2.0**-64) else _round(1 / Fraction(float(x)))
               for x in rays[i, 3:6]]
        assert [float(x) for x in got[i, :3]] == [float(x) for x in inv], i
        for c in range(8):
            t, hit = _child(rays[i], nodes[i], inv, c)
            assert (got[i, 3 + c], bool(got[i, 11 + c])) == (t, hit), (i, c)
            entered += hit
    assert n // 2 < entered < 6 * n


def _exact_mesh(n):
    """A rough height field of n x n cells, all of it in exact arithmetic
    (integers over powers of two), so the inputs are the same everywhere."""
    i, j = np.meshgrid(np.arange(n + 1), np.arange(n + 1), indexing="ij")
    k = (i * 7919 + j * 104729 + (i * j) * 31) % 1021
    x = (i * 64 + k % 37) / 256.0
    y = (j * 64 + k % 41) / 256.0
    z = ((k * k) % 509) / 4096.0
    pos = np.stack([x, y, z], -1).reshape(-1, 3).astype(f)
    v = np.arange((n + 1) * (n + 1)).reshape(n + 1, n + 1)
    a, b, c, d = v[:-1, :-1].ravel(), v[1:, :-1].ravel(), v[1:, 1:].ravel(), v[:-1, 1:].ravel()
    return pos, np.concatenate([np.stack([a, b, c], -1), np.stack([a, c, d], -1)]).astype(np.uint32)


def _edge_on(pos, tris, n, rng, far=9):
    """Rays through points of triangles' edges, nearly in the triangles'
    planes, from up to 2^far away: products, sums, quotients and square roots only (exactly rounded),
    powers of two by ldexp."""
    p = pos[tris[rng.integers(len(tris), size=n)]].astype(np.float64)
    e = p[:, 1] - p[:, 0]
    g = p[:, 2] - p[:, 0]
    x = p[:, 0] + e * (rng.integers(1, 4096, (n, 1)) / 4096.0)
    nn = np.stack([e[:, 1] * g[:, 2] - e[:, 2] * g[:, 1], e[:, 2] * g[:, 0] - e[:, 0] * g[:, 2],
                   e[:, 0] * g[:, 1] - e[:, 1] * g[:, 0]], -1)
    d = e * (rng.integers(-4096, 4096, (n, 1)) / 4096.0) + g * (rng.integers(-4096, 4096, (n, 1)) / 4096.0)
    d = d + nn * np.ldexp(rng.integers(-4096, 4096, (n, 1)) / 4096.0, -rng.integers(2, 24, (n, 1)))
    d = d / np.sqrt(d[:, :1] ** 2 + d[:, 1:2] ** 2 + d[:, 2:] ** 2)
    rays = np.zeros((n, 8), f)
    rays[:, 0:3] = x - d * np.ldexp(1.0 + rng.integers(0, 4096, (n, 1)) / 4096.0, rng.integers(-2, far, (n, 1)))
    rays[:, 3] = np.inf
    rays[:, 4:7] = d
    return rays


FAR_HITS = {False: ("82fd223b06530502", "b3775b69ddcb8179"), True: ("0fc6ef50916f092d", "3f3445fdc5cd532f")}


@pytest.mark.gpu
def test_hits_of_edge_on_rays_are_fixed():
    """Closest hits and occlusion of 2^22 edge-on rays, one value of each
    recorded when the rule was set; the form for few rays gives the same."""
    from argent_b200 import mesh as M
    from argent_b200.gpu import Context, Piece

    pos, tris = _exact_mesh(192)
    piece = Piece(Context(0), M.Mesh(pos, tris, np.zeros_like(pos), np.zeros(len(tris), np.uint16)))
    rng = np.random.default_rng(11)
    closest, occluded = hashlib.sha256(), hashlib.sha256()
    for _ in range(4):
        rays = _edge_on(pos, tris, 1 << 20, rng)
        hits, occ = piece.trace_closest(rays), piece.trace_anyhit(rays)
        closest.update(hits.tobytes())
        occluded.update(occ.tobytes())
        few = np.ascontiguousarray(rays[:8192])
        assert np.array_equal(piece.trace_closest(few).view(np.uint32), hits[:8192].view(np.uint32))
        assert np.array_equal(piece.trace_anyhit(few), occ[:8192])
    assert (closest.hexdigest()[:16], occluded.hexdigest()[:16]) == ("01f832b78b3112a0", "2e1877e372215214")


@pytest.mark.gpu
@pytest.mark.parametrize("device_bvh", [False, True])
def test_hits_of_far_rays_are_fixed(device_bvh):
    """Rays from up to 2^26 away, where a box is smaller than the interval's
    widening (more of its node's boxes are entered, absent children's inside-out
    ones too): recorded hits of both builders' trees, and the same from the form
    for few rays."""
    from argent_b200 import mesh as M
    from argent_b200.gpu import Context, Piece

    pos, tris = _exact_mesh(192)
    piece = Piece(Context(0), M.Mesh(pos, tris, np.zeros_like(pos), np.zeros(len(tris), np.uint16)),
                  device_bvh=device_bvh)
    rays = _edge_on(pos, tris, 1 << 18, np.random.default_rng(12), far=26)
    hits, occ = piece.trace_closest(rays), piece.trace_anyhit(rays)
    for k in range(0, 1 << 16, 8192):
        few = np.ascontiguousarray(rays[k:k + 8192])
        assert np.array_equal(piece.trace_closest(few).view(np.uint32), hits[k:k + 8192].view(np.uint32))
        assert np.array_equal(piece.trace_anyhit(few), occ[k:k + 8192])
    got = tuple(hashlib.sha256(a.tobytes()).hexdigest()[:16] for a in (hits, occ))
    assert got == FAR_HITS[device_bvh]
