"""The shading arithmetic that light samples use, executed: the device's own
functions compiled for the CPU (--fmad=false and IEEE division and square root,
so they round as on the device), against 64-bit values and the forms they
stand in for.  u = 2^-24 is half a unit of rounding."""

import numpy as np
import pytest

from tests import device_host

U = 2.0**-24

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "argent_b200/csrc/render_impl.cuh"
using namespace dev;
// argv: which function, floats in and out per case; cases on standard input.
int main(int argc, char** argv) {
  const std::string what = argv[1];
  const size_t ni = std::atoi(argv[2]), no = std::atoi(argv[3]);
  std::vector<float> x(ni), y(no);
  while (fread(x.data(), 4, ni, stdin) == ni) {
    if (what == "ggx") {  // alpha, wo.z, wi.z, h.z -> value and pdf, short and factor by factor
      const Ggx g{x[0]};
      const V3 wo{0, 0, x[1]}, wi{0, 0, x[2]}, h{0, 0, x[3]};
      const float lam = ggx_lambda(g, wo), d = ggx_d(g, h);
      ggx_nee(g, lam, wo, wi, h, &y[0], &y[1]);
      y[2] = d * ggx_g2(g, wo, wi) / (4.0f * wo.z * wi.z);
      y[3] = ggx_g1(g, wo) * d / wo.z / 4.0f;
    } else if (what == "conductor") {  // cos, eta, k
      y[0] = fresnel_conductor_nee(x[0], x[1], x[2]);
      y[1] = fresnel_conductor1(x[0], x[1], x[2]);
      y[2] = fresnel_conductor_normal(x[1], x[2]);
      y[3] = fresnel_conductor1(1.0f, x[1], x[2]);
    } else if (what == "coat") {  // cos, eta
      y[0] = fresnel_dielectric_nee(x[0], x[1], 1.0f / (x[1] * x[1]));
      y[1] = fresnel_dielectric(x[0], x[1]);
    } else if (what == "visible") {
      const Wavelengths w = sample_visible(x[0]);
      for (int i = 0; i < 4; ++i) y[i] = w.lambda[i], y[4 + i] = w.pdf[i];
    } else if (what == "panel") {  // centre, half axes u and v, ray o and d, reach
      DevPanel p{};
      const V3 hu{x[3], x[4], x[5]}, hv{x[6], x[7], x[8]}, n = normalize(cross(hu, hv));
      float far = 0.0f;
      for (int a = 0; a < 3; ++a) {
        p.c[a] = x[a];
        p.hu[a] = x[3 + a];
        p.hv[a] = x[6 + a];
        far += fabsf(p.c[a]) + fabsf(p.hu[a]) + fabsf(p.hv[a]);
      }
      p.n[0] = n.x;
      p.n[1] = n.y;
      p.n[2] = n.z;
      p.hu_l2 = dot(hu, hu);
      p.hv_l2 = dot(hv, hv);
      p.nd = p.n[0] * p.c[0] + p.n[1] * p.c[1] + p.n[2] * p.c[2];
      p.guard = far < 1e7f ? 3.814697265625e-06f * far : INFINITY;
      const V3 o{x[9], x[10], x[11]}, d{x[12], x[13], x[14]};
      float t;
      y[0] = panel_intersect(p, o, d, x[15], &t);
      y[1] = panel_near(p, o, d, panel_reach(o, x[15]));
    }
    fwrite(y.data(), 4, no, stdout);
  }
}
"""


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    exe = device_host.compile_program(PROGRAM, str(tmp_path_factory.mktemp("forms")))

    def call(what, no, *cols):
        x = np.stack(np.broadcast_arrays(*cols), -1).astype(np.float32)
        out = device_host.run(exe, x.tobytes(), (what, str(x.shape[1]), str(no)))
        return x.astype(np.float64).T, np.frombuffer(out, np.float32).reshape(len(x), no).T

    return call


def _errors(got, want, floor=0.0):
    e = np.abs(got.astype(np.float64) - want) / np.maximum(np.abs(want), floor)
    return e.mean(), e.max()


def test_microfacet_factors(device):
    """Ten roundings at most in each (alpha^2, k^2, two by 2 pi, lambda's four,
    the sum, the product, the quotient), each within u; and no further off than
    the factors one by one, mean and largest."""
    rng = np.random.default_rng(3)
    n = 1_500_000
    alpha = np.exp(rng.uniform(np.log(1.5e-3), 0.0, n))
    cols = alpha, rng.uniform(0.01, 1.0, n), rng.uniform(0.01, 1.0, n), np.sqrt(rng.uniform(0.2, 1.0, n))
    (a, wo, wi, _), (f, pdf, f1, pdf1) = device("ggx", 4, *cols)
    al, hz = cols[0].astype(np.float32), cols[3].astype(np.float32)
    one = np.float32(1)
    k = ((hz * hz) * (al * al - one) + one).astype(np.float64)  # D's denominator, the same in both
    lam = lambda z: 0.5 * (-1 + np.sqrt(1 + a * a * (1 - z * z) / (z * z)))  # noqa: E731
    d = a * a / (np.pi * k * k)
    want_f, want_p = d / (1 + lam(wo) + lam(wi)) / (4 * wo * wi), d / (1 + lam(wo)) / (4 * wo)
    for short, factors, want in ((f, f1, want_f), (pdf, pdf1, want_p)):
        (mean, most), (mean1, most1) = _errors(short, want), _errors(factors, want)
        assert most < 10 * U and mean <= mean1 and most <= most1, (mean, mean1, most, most1)


def test_conductor_reflectance(device):
    rng = np.random.default_rng(4)
    n = 400_000
    c = np.concatenate([rng.uniform(0.0, 1.0, n), rng.uniform(0.0, 1e-3, n // 4), [0.0, 1.0]])
    m = len(c)
    (c64, eta, k), (nee, general, normal, general1) = device("conductor", 4, c, rng.uniform(0.04, 6.0, m),
                                                             rng.uniform(0.5, 12.0, m))
    e = eta + 1j * k
    ct = np.sqrt(1 - (1 - c64 * c64) / (e * e))
    rp, rs = (e * c64 - ct) / (e * c64 + ct), (c64 - e * ct) / (c64 + e * ct)
    want = 0.5 * (np.abs(rp) ** 2 + np.abs(rs) ** 2)
    (mean, most), (mean1, most1) = _errors(nee, want), _errors(general, want)
    assert mean <= mean1 and most <= most1, (mean, mean1, most, most1)
    assert np.array_equal(normal.view(np.uint32), general1.view(np.uint32))
    # k = 0 and eta near 1: the values go to 0 at any angle but grazing ones,
    # where both forms' sin^2 is rounded away; neither is the better throughout.
    eta = np.concatenate([1.0 + rng.uniform(0.0, 1e-3, n), rng.uniform(1.0, 3.0, n), [1.0]])
    (c64, eta, _), (nee, general, normal, general1) = device("conductor", 4, rng.uniform(1e-3, 1.0, len(eta)), eta, 0.0)
    ct = np.sqrt(1 - (1 - c64 * c64) / (eta * eta))
    want = 0.5 * (((eta * c64 - ct) / (eta * c64 + ct)) ** 2 + ((c64 - eta * ct) / (c64 + eta * ct)) ** 2)
    assert np.abs(nee - want).max() <= np.abs(general - want).max()
    assert np.array_equal(normal.view(np.uint32), general1.view(np.uint32))


def test_coat_reflectance(device):
    rng = np.random.default_rng(5)
    n = 400_000
    c = np.concatenate([rng.uniform(1e-4, 1.0, n), [1.0]])
    (c64, eta), (nee, general) = device("coat", 2, c, rng.uniform(1.3, 1.8, n + 1))
    ct = np.sqrt(1 - (1 - c64 * c64) / (eta * eta))
    want = 0.5 * (((eta * c64 - ct) / (eta * c64 + ct)) ** 2 + ((c64 - eta * ct) / (c64 + eta * ct)) ** 2)
    (mean, most), (mean1, most1) = _errors(nee, want), _errors(general, want)
    assert mean <= mean1 and most <= most1, (mean, mean1, most, most1)


def test_wavelength_density(device):
    """1 - x^2 by (1 - x)(1 + x): x is off by 2 u (its product's and its own
    rounding) of at most 1.9 against 1 - |x| >= 0.029, then four roundings."""
    u = np.concatenate([np.random.default_rng(6).random(400_000), [0.0, 1.0 - U]])
    (u64,), out = device("visible", 8, u)
    lam, pdf = out[:4].astype(np.float64), out[4:].astype(np.float64)
    for i in range(4):
        up = (u64.astype(np.float32) + np.float32(i / 4)).astype(np.float32)  # as the device adds them
        up = np.where(up > 1, up - np.float32(1), up).astype(np.float64)
        x = float(np.float32(0.8569106)) - float(np.float32(1.827502)) * up
        want = float(np.float32(0.0039398042)) * (1 - x * x)
        inside = (lam[i] > 360.1) & (lam[i] < 829.9)
        assert inside.mean() > 0.99 and ((pdf[i] > 0) == ((lam[i] >= 360) & (lam[i] <= 830))).all()
        e = np.abs(pdf[i] - want)[inside] / want[inside]
        assert (e < (4 + 2 * 1.9 / (1 - np.abs(x[inside]))) * U).all()


def test_panel_test_lets_no_hit_go(device):
    """panel_near says no only where panel_intersect finds nothing, and it says
    so for a good part of the panels."""
    rng = np.random.default_rng(7)
    n = 1_000_000
    size = np.exp(rng.uniform(np.log(0.5), np.log(400.0), (n, 1)))
    hu, hv = rng.normal(size=(n, 3)), rng.normal(size=(n, 3))
    hv -= hu * (hu * hv).sum(1, keepdims=True) / (hu * hu).sum(1, keepdims=True)
    c, o = rng.normal(size=(n, 3)) * 300, rng.normal(size=(n, 3)) * 30
    at = c + hu * size * rng.uniform(-1.1, 1.1, (n, 1)) + hv * size * rng.uniform(-1.1, 1.1, (n, 1))
    d = np.where(rng.random((n, 1)) < 0.6, at - o, rng.normal(size=(n, 3)))
    dist = np.linalg.norm(d, axis=1, keepdims=True)
    d /= dist
    # Reaches that end near the panel's plane, beyond it, and never.
    t = np.where(rng.random((n, 1)) < 0.5, dist * (1 + rng.normal(size=(n, 1)) * 10.0 ** rng.uniform(-7, 0, (n, 1))),
                 np.where(rng.random((n, 1)) < 0.5, np.inf, rng.uniform(0, 1000, (n, 1))))
    x = np.hstack([c, hu * size, hv * size, o, d, t])
    _, (hit, near) = device("panel", 2, *x.T)
    assert not ((hit == 1) & (near == 0)).any()
    assert hit.sum() > n // 10 and (near == 0).sum() > 0.3 * (hit == 0).sum()
