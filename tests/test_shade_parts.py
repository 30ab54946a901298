"""A film does not depend on which shade kernels drew it: waves below and from 2 Mi paths on
(hits and misses apart), and batches whose scenes need more code than one of them does."""
import numpy as np
import pytest

from luz_b200 import native, scenes

pytestmark = pytest.mark.gpu

CASES = {
    "glossy": lambda: scenes.mesh_glossy(256, 256, 40, 8, level=5),
    "cornell": lambda: scenes.cornell(256, 256, 40, 8),
    "spheres": lambda: scenes.spheres_linear_sky(256, 256, 40, 8),
    "instances": lambda: scenes.instancing_volumes(256, 256, 40, 6, count=300),
    "mixed": lambda: scenes.tiny_mixed(256, 256, 40, 6),
    "atmosphere": lambda: scenes.atmosphere_hills(256, 256, 40, 3),
    "caustics": lambda: scenes.caustic_pool(256, 256, 40, 6, photons=4000),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_the_film_does_not_depend_on_the_wave_size(name):
    w = CASES[name]()
    g = native.GpuScene(w.scene.build())
    try:
        p = native.params(w.width, w.height, w.spp, w.max_bounces, 11)
        whole, s0 = g.render(p)                # one wave of 2.6 M paths
        g.set_tuning(wave_paths=1 << 20)
        parts, s1 = g.render(p)                # waves below 2 Mi paths
        assert s0.waves == 1 and s1.waves == 3
        assert np.array_equal(whole, parts), int((whole != parts).any(-1).sum())
        assert (s0.extension_rays, s0.shadow_rays) == (s1.extension_rays, s1.shadow_rays)
    finally:
        g.close()


@pytest.mark.parametrize("beside", ["mixed", "ies", "caustics"])
def test_a_batch_mate_does_not_change_a_film(beside):
    """Beside a scene with Principled materials, IES lights or caustics a plain scene is shaded
    by the kernels with that code: the film is its own render's."""
    mate = {"mixed": scenes.tiny_mixed(32, 24, 2, 4), "ies": scenes.ies_room(32, 24, 2, 4),
            "caustics": scenes.caustic_pool(32, 24, 2, 4, photons=2000)}[beside]
    ws = [scenes.mesh_glossy(160, 120, 24, 8, level=5), scenes.cornell(120, 120, 24, 8),
          scenes.spheres_linear_sky(128, 96, 24, 8), mate]
    gs = [native.GpuScene(w.scene.build()) for w in ws]
    try:
        ps = [native.params(w.width, w.height, w.spp, w.max_bounces, 5 + i) for i, w in enumerate(ws)]
        films, _ = native.batch_render(gs, ps)
        for w, g, p, film in zip(ws, gs, ps, films):
            own, _ = g.render(p)
            assert np.array_equal(film, own), (w.name, int((film != own).any(-1).sum()))
    finally:
        for g in gs:
            g.close()
