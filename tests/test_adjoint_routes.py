"""Which passes a texture gradient runs, read off its launches.

A trace of a wave with B bounces launches ray generation once, the trace stage B + 2 times and
the shade stage B + 1 times, in one launch each: the gradient kernels shade hits and misses
together at every wave size."""
import numpy as np
import pytest

from luz_b200 import native, scenes

pytestmark = pytest.mark.gpu


def trace_launches(bounces: int) -> int:
    return 1 + (bounces + 2) + (bounces + 1)


@pytest.mark.parametrize("side,spp", [(9, 5), (40, 8)])
def test_more_visits_than_records_take_two_traces(side, spp):
    """A closed room with one texture on every wall: more visits than there are records, so the
    recording trace gives the paths' radiance (one launch adds it up) and a replay the gradient."""
    bounces = 3
    w = scenes.cornell(side, side, spp, bounces, closed=True)
    s = w.scene
    texels = np.random.default_rng(5).uniform(0.4, 0.6, (8, 8, 3))
    t = s.texture(texels)
    m = s.lambertian((1.0, 1.0, 1.0), texture=t)
    for o in s.objects:
        if s.materials[o["material"]]["type"] == 1:
            o["material"] = m
    g = native.GpuScene(s.build())
    try:
        adj = np.ones((side, side, 3), np.float32)
        grad, st = g.adjoint_backward(native.params(side, side, spp, bounces, 17), t, adj, texels.shape)
        assert np.abs(grad).sum() > 0.0 and st.waves == 1
        assert st.kernel_launches == 2 * trace_launches(bounces) + 1, st.kernel_launches
    finally:
        g.close()


@pytest.mark.parametrize("side,spp", [(24, 3), (256, 32)])
def test_roughness_passes_run_the_same_kernels(side, spp):
    """Pass one fixes each path's radiance, pass two replays the path: both run the same shade
    kernel (another one may round a decision otherwise), on waves below and from 2 Mi paths on."""
    bounces = 2
    w = scenes.cornell_rough_panel(side, side, spp, bounces)
    g = native.GpuScene(w.scene.build())
    try:
        adj = np.ones((side, side, 3), np.float32)
        grad, st = g.adjoint_backward(native.params(side, side, spp, bounces, 3), 1, adj, (64, 64, 3))
        assert np.abs(grad).sum() > 0.0 and st.waves == 1
        assert st.kernel_launches == 2 * trace_launches(bounces) + 2, st.kernel_launches
    finally:
        g.close()


def test_recorded_visits_count_against_the_budget():
    """A path takes 276 bytes of state and two records of 24 bytes: a budget of 4,096 paths'
    state and records makes sixteen waves of 65,536 paths (fourteen if the state alone counted),
    and the same gradient."""
    side, spp, bounces = 128, 4, 3
    w = scenes.cornell_textured(side, side, spp, bounces)
    g = native.GpuScene(w.scene.build())
    try:
        p = native.params(side, side, spp, bounces, 9)
        adj = np.random.default_rng(2).uniform(0.5, 1.5, (side, side, 3)).astype(np.float32)
        ref, s0 = g.adjoint_backward(p, 0, adj, (32, 32, 3))
        g.set_path_budget((276 + 48) * 4096)
        got, s1 = g.adjoint_backward(p, 0, adj, (32, 32, 3))
        assert s0.waves == 1 and s1.waves == side * side * spp // 4096, (s0.waves, s1.waves)
        assert np.allclose(got, ref, rtol=1e-12, atol=1e-18)
    finally:
        g.close()
