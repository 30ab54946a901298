"""The albedo-texture gradient by both of its routes (one pass that records the paths' visits
of the texture, and the two passes a wave takes when it has more than two visits per path)
against central differences of the film in a common factor of all texels.

Up to bounce 3 nothing but the throughput depends on the albedo, so the film is a polynomial
of degree at most 5 in the factor: with h = 2e-3 a central difference is off by less than
(5 choose 3) h^2 = 4e-5 relative, and the film's FP32 rounding (6e-8) adds 6e-8 / 2h = 1.5e-5:
below 1e-3 together, which also leaves room for the pixels' sums."""
import numpy as np
import pytest

from luz_b200 import native, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("walls,per_path", [(1, "at most two"), (6, "more than two")])
@pytest.mark.parametrize("side,spp", [(1, 1), (9, 5), (40, 8)])
def test_albedo_gradient_against_differences(walls, per_path, side, spp):
    w = scenes.cornell(side, side, spp, 3, closed=True)
    s = w.scene
    texels = np.random.default_rng(walls).uniform(0.4, 0.6, (8, 8, 3))
    t = s.texture(texels)
    m = s.lambertian((1.0, 1.0, 1.0), texture=t)
    white = [o for o in s.objects if o["kind"] == 1 and s.materials[o["material"]]["type"] == 1]
    for o in white[:1] if walls == 1 else s.objects:
        if s.materials[o["material"]]["type"] == 1:
            o["material"] = m
    g = native.GpuScene(s.build())
    try:
        p = native.params(side, side, spp, 3, 17)
        adj = np.random.default_rng(3).uniform(0.5, 1.5, (side, side, 3)).astype(np.float32)
        grad, _ = g.adjoint_backward(p, t, adj, texels.shape)
        again, _ = g.adjoint_backward(p, t, adj, texels.shape)
        assert np.allclose(grad, again, rtol=1e-12, atol=0.0)
        h = 2e-3

        def film(k):
            return float(np.sum(g.adjoint_forward(p, t, texels * k)[0].astype(np.float64) * adj))

        want = (film(1.0 + h) - film(1.0 - h)) / (2.0 * h)
        got = float(np.sum(grad * texels))
        assert abs(got - want) <= 1e-3 * max(abs(want), 1e-6), (got, want, per_path)
    finally:
        g.close()
