"""The lane-in-step traversal (walk.cuh) against the FP32 restatement, bit for bit, where
its own rules decide: leaves of every size (grouped and per-lane triangle tests), equal
distances (every triangle twice, rays through shared vertices and edges), the skip of an
empty slot, instances entered and left, top-level leaves of four and more children, and
ray counts around a warp and a block. The collapsed nodes are checked on the CPU against
the binary ones they stand for."""
import numpy as np
import pytest

from luz_b200 import native, scenes
from luz_b200.desc import Scene

NODE = np.dtype([("lmin", "<f4", 3), ("lmax", "<f4", 3), ("rmin", "<f4", 3), ("rmax", "<f4", 3),
                 ("lref", "<u4"), ("rref", "<u4"), ("pad", "<u4", 2)])
NODE4 = np.dtype([("lo", "<f4", (3, 4)), ("ref", "<u4", 4), ("hi", "<f4", (3, 4)), ("pad", "<u4", 4)])
LEAF, EMPTY, EMPTY_PLANE = 0x80000000, 0xFFFFFFFF, np.float32(3.0e38)


def soup(n: int, seed: int) -> np.ndarray:
    """n triangles on a coarse lattice (shared corners and edges), the odd ones repeated."""
    rng = np.random.default_rng(seed)
    k = int(np.ceil(n ** (1.0 / 3.0))) + 1
    t = (rng.integers(0, k, (n, 1, 3)) + rng.integers(0, 2, (n, 3, 3))).astype(np.float64)
    flat = np.linalg.norm(np.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0]), axis=1) == 0
    t[flat] = t[flat][:, :1] + np.eye(3)[None]
    t[1::2] = t[:2 * (n // 2):2]
    return t / k


def scene(n: int, instances: bool, seed: int) -> Scene:
    s = Scene()
    white = s.lambertian((0.7, 0.7, 0.7))
    s.background = (0.1, 0.1, 0.1)
    m, _ = s.mesh(soup(n, seed), white)
    if instances:
        for j in range(9):
            s.mesh_instance(m, (0.3 * j - 1.0, 0.1 * (j % 2), 0.2), (10.0 * j, 20.0 * (j % 3), 0.0),
                            (1.0, 1.0 + 0.25 * (j % 2), 0.8), white)
        s.rectangle((0.5, 0.5, -0.4), (0, 0, 1), 3.0, 3.0, white)
        s.sphere((0.5, 0.5, 0.5), 0.2, white)
        s.volume_sphere((0.2, 0.2, 0.2), 0.6, s.isotropic((0.5, 0.5, 0.5)), 0.4)
    return s


def rays(n: int, tris: np.ndarray, seed: int) -> np.ndarray:
    """Half of the rays aim at corners and edge midpoints from lattice points, half at random."""
    rng = np.random.default_rng(seed)
    aim = tris[rng.integers(0, len(tris), n), rng.integers(0, 3, n)]
    other = tris[rng.integers(0, len(tris), n), rng.integers(0, 3, n)]
    aim = np.where(rng.random((n, 1)) < 0.5, aim, 0.5 * (aim + other))
    org = rng.integers(-2, 4, (n, 3)).astype(np.float64)
    rand = rng.random((n, 1)) < 0.5
    org = np.where(rand, rng.normal(0.5, 1.5, (n, 3)), org)
    d = np.where(rand, rng.normal(0.5, 0.4, (n, 3)), aim) - org
    d[np.linalg.norm(d, axis=1) == 0] = (0.0, 0.0, 1.0)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3], r[:, 3], r[:, 4:7], r[:, 7] = org, 1e-3, d, np.where(rng.random(n) < 0.8, np.inf, 1.0)
    return r


@pytest.mark.parametrize("n", [1, 8, 9, 33, 700, 5000])
def test_collapsed_nodes_hold_the_binary_trees_boxes(n):
    pk = native.Pack(scene(n, False, n).build())
    nodes, nodes4 = pk.array("mesh_nodes").view(NODE), pk.array("mesh_nodes4").view(NODE4)
    if len(nodes) == 0:
        assert len(nodes4) == 0
        return
    at, stack = 0, [(0, 0)]   # (binary node, collapsed node); the root is the first of both
    while stack:
        b, q = stack.pop()
        at += 1
        for side, (ref, mn, mx) in enumerate((("lref", "lmin", "lmax"), ("rref", "rmin", "rmax"))):
            r = int(nodes[b][ref])
            lo, hi = nodes4[q]["lo"][:, 2 * side:2 * side + 2], nodes4[q]["hi"][:, 2 * side:2 * side + 2]
            assert np.array_equal(lo.min(1), nodes[b][mn]) and np.array_equal(hi.max(1), nodes[b][mx])
            refs = nodes4[q]["ref"][2 * side:2 * side + 2]
            if r & LEAF:
                assert refs[0] == r and refs[1] == EMPTY and (lo[:, 1] == EMPTY_PLANE).all() and (hi[:, 1] == -EMPTY_PLANE).all()
                continue
            for k, (gref, gmn, gmx) in enumerate((("lref", "lmin", "lmax"), ("rref", "rmin", "rmax"))):
                g = int(nodes[r][gref])
                assert np.array_equal(lo[:, k], nodes[r][gmn]) and np.array_equal(hi[:, k], nodes[r][gmx])
                if g & LEAF:
                    assert refs[k] == g
                else:
                    stack.append((g, int(refs[k])))
    assert at == len(nodes4)


@pytest.mark.gpu
@pytest.mark.parametrize("instances", [False, True])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 33, 700, 5000])
def test_walk_equals_the_restatement(n, instances, restate):
    s = scene(n, instances, n)
    b = s.build()
    pk, g = native.Pack(b), native.GpuScene(b)
    try:
        for count in (1, 31, 33, 129, 4001):
            r = rays(count, np.asarray(s.meshes[0]["positions"]).reshape(-1, 3, 3), seed=n + count)
            key = np.stack([np.arange(count), np.arange(count) * 7, np.arange(count) % 5, np.arange(count) % 3], 1).astype(np.int32)
            for any_hit in (False, True):
                got = g.trace_rays(r, any_hit=any_hit, seed=3, volume_key=key)
                want = restate.trace(pk, r, any_hit=any_hit, seed=3, volume_key=key)
                assert got.tobytes() == want.tobytes(), (count, any_hit, np.flatnonzero(got != want)[:5])
    finally:
        g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("side", [1, 3, 8, 11])
def test_short_queues_give_the_same_paths_as_long_ones(side):
    """A wave of few paths spreads its rays thinly over the warps; its paths equal those of
    the same pixels inside a frame that fills them."""
    w = scenes.mesh_glossy(96, 96, 4, 8, level=4)
    g = native.GpuScene(w.scene.build())
    try:
        p = native.params(96, 96, 4, 8, w.seed)
        film, _ = g.render(p)
        y, x = np.divmod(np.arange(side * side), side)
        few, _ = g.render_pixels(p, x + 40, y + 40)
        assert np.array_equal(few.reshape(side, side, 3), film[40:40 + side, 40:40 + side])
    finally:
        g.close()
