"""NFOR's regression kernels at their edges (tiles cut by the image, windows as wide as a tile
holds and wider, buffers with values that are not finite) against a numpy restatement of
Denoise::applyNFOR (NFOR.cpp:977-1102) that solves each pixel's normal equations with LAPACK.

The systems are symmetric, with a ridge of 1e-4 and entries of at most K (the window's pixel
count, 225 here), so their condition number is below 1e7; FP64 rounding (1.1e-16) of either
solver then moves a result by about 1e-9 relative at most, and two solvers agree to 1e-8."""
import numpy as np
import pytest

from luz_b200 import native

RIDGE, LUM = 1e-4, np.array([0.2722287168, 0.6740817658, 0.0536895174])


def shifts(radius):
    return [(dy, dx) for dy in range(-radius, radius + 1) for dx in range(-radius, radius + 1)]


def at(img, dy, dx):
    """img at (y + dy, x + dx), coordinates clamped."""
    h, w = img.shape[:2]
    return img[np.clip(np.arange(h) + dy, 0, h - 1)][:, np.clip(np.arange(w) + dx, 0, w - 1)]


def patch_distance(img, var, scale, dy, dx, patch, minvar):
    h, w = img.shape[:2]
    ys, xs = np.clip(np.arange(h) + dy, 0, h - 1), np.clip(np.arange(w) + dx, 0, w - 1)
    d, n = np.zeros((h, w)), 0
    for py, px in shifts(patch):
        ay, ax = np.clip(np.arange(h) + py, 0, h - 1), np.clip(np.arange(w) + px, 0, w - 1)
        by, bx = np.clip(ys + py, 0, h - 1), np.clip(xs + px, 0, w - 1)
        a, b = img[ay][:, ax], img[by][:, bx]
        d += np.sum((a - b) ** 2, -1) / 3.0 / (var[ay][:, ax] * scale + var[by][:, bx] * scale + minvar)
        n += 1
    same = (ys == np.arange(h))[:, None] & (xs == np.arange(w))[None, :]
    return np.where(same, 0.0, d / n)


def regression(img, feats, var, scale, radius, patch, bw, minvar):
    h, w = img.shape[:2]
    m = np.zeros((h, w, 12, 12)) + RIDGE * np.eye(12)
    rhs = np.zeros((h, w, 12, 3))
    for dy, dx in shifts(radius):
        wgt = np.exp(-patch_distance(img, var, scale, dy, dx, patch, minvar) / max(minvar, bw * bw))
        b = np.concatenate([np.ones((h, w, 1)), at(feats, dy, dx) - feats], -1)
        m += wgt[..., None, None] * b[..., :, None] * b[..., None, :]
        rhs += wgt[..., None, None] * b[..., :, None] * at(img, dy, dx)[..., None, :]
    return np.linalg.solve(m, rhs)[..., 0, :]


def nfor(b, prefilter, radius, patch, minvar):
    """applyNFOR for images without fireflies (every luminance below 0.30)."""
    ca, cb, cv, fa, fb, fv = (b[k] for k in ("color_a", "color_b", "color_variance", "features_a", "features_b",
                                             "feature_variance"))
    assert (np.nan_to_num(ca) @ LUM).max() < 0.3 and (np.nan_to_num(cb) @ LUM).max() < 0.3

    def pre(img, guide):
        avg, s = fv.mean(-1), max(1.0, float(prefilter))
        acc, tot = np.zeros_like(img), np.zeros(img.shape[:2])
        for dy, dx in shifts(prefilter):
            d = np.mean((guide - at(guide, dy, dx)) ** 2, -1) / (avg + at(avg, dy, dx) + minvar)
            wgt = np.exp(-d / 0.25) * np.exp(-(dx * dx + dy * dy) / (2.0 * s * s))
            acc += at(img, dy, dx) * wgt[..., None]
            tot += wgt
        return acc / tot[..., None]

    col, pa, pb = (ca + cb) * 0.5, pre(fa, fb), pre(fb, fa)
    ra = [regression(ca, pb, cv, 2.0, radius, patch, bw, minvar) for bw in (0.5, 1.0)]
    rb = [regression(cb, pa, cv, 2.0, radius, patch, bw, minvar) for bw in (0.5, 1.0)]
    dist = lambda p, q: np.sum((p - q) ** 2, -1) / 3.0

    def mse(x, y):
        v = (dist(cb, x) - 4.0 * cv + dist(ca, y) - 4.0 * cv) * 0.5 - dist(x, y) * 0.25
        return np.where(v > 0.0, v, 0.0)

    def pair(p, q):
        sp, sq, tot = np.zeros_like(p), np.zeros_like(q), np.zeros_like(p)
        for dy, dx in shifts(3):
            wgt = np.exp(-patch_distance(col, cv, 1.0, dy, dx, 1, minvar) / max(minvar, 1.0))
            sp += at(p, dy, dx) * wgt
            sq += at(q, dy, dx) * wgt
            tot += wgt
        return sp / tot, sq / tot

    m1, m2 = pair(mse(ra[0], rb[0]), mse(ra[1], rb[1]))
    s1, s2 = pair((m1 <= m2).astype(float), (m2 <= m1).astype(float))
    st = s1 + s2
    w0 = np.where(st > minvar, s1 / np.where(st > minvar, st, 1.0), (m1 <= m2).astype(float))[..., None]
    comb = ((ra[0] * w0 + ra[1] * (1.0 - w0)) + (rb[0] * w0 + rb[1] * (1.0 - w0))) * 0.5
    return regression(comb, pa * 0.5 + pb * 0.5, dist(ra[1], rb[1]) * 0.25, 1.0, radius, patch, 1.0, minvar)


def buffers(w, h, seed):
    rng = np.random.default_rng(seed)
    f = rng.random((h, w, 11))
    ca = 0.2 * rng.random((h, w, 3))
    cb = np.clip(ca + 0.02 * rng.normal(size=ca.shape), 0.0, 0.25)
    return {"color_a": ca, "color_b": cb, "color_variance": 1e-4 + 1e-3 * rng.random((h, w)), "features_a": f,
            "features_b": f + 0.02 * rng.normal(size=f.shape), "feature_variance": 1e-4 + 1e-3 * rng.random((h, w, 11))}


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,radius", [(1, 1, 2), (2, 3, 1), (16, 2, 2), (17, 9, 2), (33, 5, 4), (31, 7, 5), (20, 18, 6),
                                        (18, 17, 7), (64, 9, 3), (65, 8, 2)])
def test_regression_equals_the_restatement(w, h, radius):
    b = buffers(w, h, 10 * w + h)
    out = native.nfor_denoise(b, regression_radius=radius)
    want = nfor(b, 1, radius, 1, 1e-5)
    assert np.allclose(out, want, rtol=1e-8, atol=1e-10), np.abs(out - want).max()


@pytest.mark.gpu
def test_values_that_are_not_finite_stay_near_their_pixel():
    """A NaN feature spoils the systems that read it (prefilter, two regressions, the filters of
    the selection: 1 + 2 + 3 + 3 + 1 + 2 pixels away at most) and no other."""
    b = buffers(40, 36, 5)
    clean = native.nfor_denoise(b)
    b["features_a"] = b["features_a"].copy()
    b["features_a"][4, 6, 3] = np.nan
    out = native.nfor_denoise(b)
    assert not np.isfinite(out[4, 6]).any()
    far = np.ones((36, 40), bool)
    far[:4 + 13, :6 + 13] = False
    assert np.array_equal(out[far], clean[far])
