"""Short forms of the shading arithmetic, restated operation by operation in
float32 (numpy rounds each operation as the device does; a fused
multiply-add is one rounding of the float64 value) and compared with the
general forms they stand in for."""

import numpy as np

f = np.float32


def fma(a, b, c):
    return (np.float64(1) * a * b + c).astype(f)


def fresnel_conductor1(c, eta, k):
    """spectral.cuh fresnel_conductor1 (fresnel.rs:81-93)."""
    c = np.clip(c, f(0), f(1))
    s2 = f(1) - c * c
    er, ei = eta * eta - k * k, eta * k + k * eta
    dd = er * er + ei * ei
    sr, si = (s2 * er + f(0) * ei) / dd, (f(0) * er - s2 * ei) / dd
    ar, ai = f(1) - sr, f(0) - si
    n = np.sqrt(ar * ar + ai * ai)
    t1 = np.sqrt(f(0.5) * (n + np.abs(ar)))
    t2 = f(0.5) * ai / t1
    cr, ci = np.where(ar >= 0, t1, np.abs(t2)), np.where(ar >= 0, t2, np.copysign(t1, ai))

    def ratio(nr, ni, dr, di):
        d = dr * dr + di * di
        return (nr * dr + ni * di) / d, (ni * dr - nr * di) / d

    pr, pi = ratio(eta * c - cr, k * c - ci, eta * c + cr, k * c + ci)
    xr, xi = eta * cr - k * ci, eta * ci + k * cr
    rr, ri = ratio(c - xr, f(0) - xi, c + xr, f(0) + xi)
    return f(0.5) * ((pr * pr + pi * pi) + (rr * rr + ri * ri))


def test_normal_incidence_rounds_as_the_general_form():
    rng = np.random.default_rng(5)
    n = 500_000
    eta = np.concatenate([rng.uniform(0.02, 6.0, n), [0.05, 1.0, 1.5, 1.0]]).astype(f)
    k = np.concatenate([rng.uniform(0.0, 12.0, n), [0.0, 0.0, 0.0, 5.0]]).astype(f)
    nr, dr = eta - f(1), eta + f(1)
    dd = dr * dr + k * k
    a, b = (nr * dr + k * k) / dd, (k * dr - nr * k) / dd
    short = a * a + b * b
    assert np.array_equal(short, fresnel_conductor1(np.ones_like(eta), eta, k))


def panel_intersect(n, c, hu, hv, hu2, hv2, o, d, t_max):
    """render_impl.cuh panel_intersect (light.rs:50-63): hit or not."""
    dot = lambda a, b: (a[0] * b[0] + a[1] * b[1]) + a[2] * b[2]  # noqa: E731
    den = dot(d, n)
    num = dot([c[i] - o[i] for i in range(3)], n)
    ok = (np.abs(den) >= f(1e-9)) & (num != 0) & (np.signbit(num) == np.signbit(den))
    with np.errstate(all="ignore"):
        t = num / den
        ok &= (t > f(1e-6)) & (t < t_max)
        q = [(o[i] + d[i] * t) - c[i] for i in range(3)]
        return ok & (np.abs(dot(q, hu) / hu2) <= 1) & (np.abs(dot(q, hv) / hv2) <= 1)


def panel_near(n, nd, guard, o, d, t_max):
    """render_impl.cuh panel_reach and panel_near."""
    u = f(2.0**-18)
    t = np.minimum(t_max, f(1e8))
    om = (np.abs(o[0]) + np.abs(o[1])) + np.abs(o[2])
    m = np.where(om < f(1e7), u * (om + t), f(np.inf)).astype(f) + guard
    s = fma(-n[2], o[2], fma(-n[1], o[1], fma(-n[0], o[0], nd)))
    den = fma(n[2], d[2], fma(n[1], d[1], n[0] * d[0]))
    e = fma(-t, den, s)
    return ~((np.minimum(s, e) > m) | (np.maximum(s, e) < -m))


def test_panel_near_keeps_every_hit():
    """Panels of 1e-2 to 1e5 mm at 1 to 1e6 mm, rays aimed into, past, away
    from and along them, segments that end just short of and just past them
    and rays without an end: whatever panel_intersect hits, panel_near keeps,
    and it lets most segments that do not cross the plane go."""
    rng = np.random.default_rng(9)
    let_go = total = 0
    for size in (1e-2, 1.0, 30.0, 1e3, 1e5):
        for far in (1.0, 60.0, 1e4, 1e6):
            m = 20_000
            unit = lambda: (lambda v: v / np.linalg.norm(v, axis=0))(rng.normal(size=(3, m)))  # noqa: E731
            n64 = unit()
            a = np.cross(n64, unit(), axis=0)
            a /= np.linalg.norm(a, axis=0)
            b = np.cross(n64, a, axis=0)
            c64 = unit() * far
            hu, hv = (a * size).astype(f), (b * size * rng.uniform(0.1, 1.0, m)).astype(f)
            c = c64.astype(f)
            w = np.cross(hu.astype(np.float64), hv, axis=0)
            n = (w / np.linalg.norm(w, axis=0)).astype(f)
            hu2, hv2 = ((h[0] * h[0] + h[1] * h[1]) + h[2] * h[2] for h in (hu, hv))
            o = (unit() * rng.uniform(0.0, 40.0, m)).astype(f)
            aim = c + hu * rng.uniform(-1.5, 1.5, m).astype(f) + hv * rng.uniform(-1.5, 1.5, m).astype(f)
            d64 = aim.astype(np.float64) - o
            dist = np.linalg.norm(d64, axis=0)
            d64 = np.where(rng.random(m) < 0.3, unit(), d64 / dist)  # some anywhere
            d64 = np.where(rng.random(m) < 0.1, a, d64)  # some along the plane
            d = (d64 / np.linalg.norm(d64, axis=0)).astype(f)
            t_max = np.choose(rng.integers(0, 4, m), [dist * 0.9999, dist * 1.0001, dist * rng.uniform(0.1, 3.0, m),
                                                      np.full(m, np.inf)]).astype(f)
            nd = (n[0] * c[0] + n[1] * c[1]) + n[2] * c[2]
            span = sum(np.abs(x).sum(0) for x in (c, hu, hv)).astype(f)
            guard = np.where(span < f(1e7), f(2.0**-18) * span, f(np.inf)).astype(f)
            hit, near = panel_intersect(n, c, hu, hv, hu2, hv2, o, d, t_max), panel_near(n, nd, guard, o, d, t_max)
            assert not (hit & ~near).any(), (size, far)
            let_go += int((~near).sum())
            total += int((~hit).sum())
    assert let_go > 0.3 * total
