"""The walk with rays that are no rays (origins and directions that are not numbers, infinite,
or near the ends of FP32) against the FP32 restatement, bit for bit."""
import numpy as np
import pytest

from luz_b200 import native
from test_walk import rays, scene


def extreme_rays(n: int, tris: np.ndarray, seed: int) -> np.ndarray:
    rng = np.random.default_rng(seed)
    r = rays(n, tris, seed)   # (an interval that is no number leaves no answer to hold the walk to)
    odd = np.array([np.nan, np.inf, -np.inf, 3.0e38, -3.0e38, 1.0e-38, -1.0e-45, 0.0, -0.0, 4095.9, 4096.0], np.float32)
    for i in range(n):
        k = rng.integers(0, 4)
        for cols in ([(0, 1, 2)], [(4, 5, 6)], [(0, 1, 2), (4, 5, 6)], [(3, 7)])[k]:   # origin, direction, both, interval
            hit = [c for c in cols if rng.random() < 0.5] or [cols[0]]
            r[i, hit] = rng.choice(odd[1:] if k == 3 else odd, len(hit))
    return r


def test_no_ray_meets_an_empty_slot():
    """The fast box form on an empty slot's inverted box, over every combination of component
    values the form accepts (finite non-zero inverse directions, the largest finite origin
    component below 4096): rejected, so the slot's reference is never followed. FP32 FMA from
    exact FP64 products; max and min pass over a NaN, as the device's do."""
    one = np.float32
    with np.errstate(all="ignore"):
        d = np.concatenate([v * s for s in (1, -1) for v in [np.array(
            [1e-45, 1e-40, 2e-39, 3e-39, 1.2e-38, 1e-30, 1e-3, 0.5, 1, 7, 1e10, 1e30, 8.5e37, 1e38, 3.4e38], one)]])
        inv = one(1) / d
        inv = inv[np.isfinite(inv) & (inv != 0)]
        o = np.array([0, -0.0, 1e-45, 1, -1, 17.5, -333, 4095.99, -4095.99, np.nan], one)
        I, O = (a.ravel() for a in np.meshgrid(inv, o))
        noi = -(O * I)

        def fma(plane):   # the product of two FP32 values is exact in FP64
            return (np.float64(plane) * I.astype(np.float64) + noi.astype(np.float64)).astype(one)

        lo, hi = fma(one(3e38)), fma(one(-3e38))
        near, far = np.where(I > 0, lo, hi), np.where(I > 0, hi, lo)
        near, far = np.fmax(one(1e-3), near), np.fmin(one(np.inf), far)
        finite = ~np.isnan(O)
        # one finite component rejects, whatever the others' NaNs leave of the interval
        assert (far[finite] <= near[finite]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("instances", [False, True])
@pytest.mark.parametrize("n", [1, 9, 700])
def test_extreme_rays_equal_the_restatement(n, instances, restate):
    s = scene(n, instances, n)
    b = s.build()
    pk, g = native.Pack(b), native.GpuScene(b)
    try:
        r = extreme_rays(6007, np.asarray(s.meshes[0]["positions"]).reshape(-1, 3, 3), seed=n)
        for any_hit in (False, True):
            got = g.trace_rays(r, any_hit=any_hit, seed=3)
            want = restate.trace(pk, r, any_hit=any_hit, seed=3)
            number = ~np.isnan(want["t"])
            assert got[number].tobytes() == want[number].tobytes(), any_hit
            # distances that are no numbers have no order: one of the ray's hits is reported
            odd = got[~number]
            assert np.isnan(odd["t"]).all() and (odd["object"] >= 0).all() and (odd["primitive"] >= 0).all()
            assert (odd["object"] < max(1, len(s.objects))).all() and (odd["primitive"] < max(6, n)).all()
    finally:
        g.close()
