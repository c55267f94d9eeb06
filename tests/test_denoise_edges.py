"""The device denoiser at sizes where its tiles (32 x 8 pixels) and taps (up
to 32 pixels apart) leave the image: against the oracle's atrous, which
differs by expf alone (1e-4 of the largest value, as tests/test_denoise.py
allows)."""

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(1, 1), (1, 40), (3, 2), (31, 9), (33, 7), (64, 8), (65, 17), (200, 131)])
@pytest.mark.parametrize("guides", [0, 1, 2])
def test_denoise_at_tile_edges(w, h, guides):
    import oracle as O
    from argent_b200 import gpu as G

    rng = np.random.default_rng(1000 * w + h)
    color = np.exp(rng.normal(size=(h, w, 3))).astype(np.float32)
    albedo = rng.uniform(0.0, 1.1, (h, w, 3)).astype(np.float32)
    normal = rng.normal(size=(h, w, 3)).astype(np.float32)
    normal /= np.linalg.norm(normal, axis=-1, keepdims=True)
    normal[rng.random((h, w)) < 0.1] = 0.0
    color[0, 0] = [np.nan, -1.0, np.inf]
    a = albedo if guides >= 1 else None
    n = normal if guides >= 2 else None
    ctx = G.Context(0)
    got = G.denoise_atrous(ctx, color, a, n)
    want = O.atrous(color, a, n)
    assert np.isfinite(want).all()
    assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max()
