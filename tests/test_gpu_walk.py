"""The walk against brute force: every voxel's box test (box_test,
primitives.glsl:273-355) in numpy single precision, in the kernels' operation
order, decides each ray's closest hit and visibility.  The scenes lie at the
edges of what the walk indexes: a single voxel, rows of up to 1024 cells on
each axis, negative coordinates, voxel edges that are and are not powers of
two; the rays run along axes and diagonals, start inside voxels and on their
faces, and cover every octant."""
import numpy as np
import pytest

from cube_tracing import layouts as L
from cube_tracing import scenes

F = np.float32


def line_scene(cells, extent=1.0):
    """A scene of the given integer cells (no lights)."""
    c = np.asarray(cells, np.int64)
    sc = scenes._build(c, np.zeros(len(c), bool), np.full((1, 3), 0.5, F), np.zeros(len(c), np.uint32),
                       np.zeros((0, 3), F), extent, (1, 1, 1), "line", {})
    return sc


def scene(name):
    rng = np.random.default_rng(3)
    if name == "one":
        return line_scene([(0, 0, 0)])
    if name in ("row_x", "row_y", "row_z"):
        a = "xyz".index(name[-1])
        c = np.zeros((40, 3), np.int64)
        c[:, a] = np.sort(rng.choice(1014, 40, replace=False))
        c[0, a], c[-1, a] = 0, 1013
        return line_scene(c)
    if name == "negative":
        return line_scene(np.unique(rng.integers(-21, -3, (300, 3)), axis=0))
    extent = {"grid": 1.0, "edge5": 2.0 ** -5, "edge03": 0.3}[name]
    return line_scene(np.unique(rng.integers(0, 13, (400, 3)), axis=0), extent)


def ray_set(sc, n, seed):
    rng = np.random.default_rng(seed)
    lo, hi = sc.aabbs["minimum"].min(0), sc.aabbs["maximum"].max(0)
    pad = 3 * sc.voxel_extent
    o = rng.uniform(lo - pad, hi + pad, (n, 3)).astype(F)
    pick = sc.aabbs[rng.integers(0, sc.voxel_count, n)]
    at = (pick["minimum"] + (pick["maximum"] - pick["minimum"]) * rng.choice([0.0, 0.25, 0.5, 1.0], (n, 3))).astype(F)
    d = (at - o).astype(F)
    flat = rng.random(n) < 0.3  # along an axis or a diagonal, from a voxel's corner, face or inside
    d[flat] = rng.integers(-1, 2, (int(flat.sum()), 3)).astype(F)
    o[flat] = at[flat] - d[flat] * F(sc.voxel_extent) * rng.choice([0, 1, 2, 3], (int(flat.sum()), 1)).astype(F)
    d[(d == 0).all(1)] = (1, 0, 0)
    d = (d / np.sqrt((d * d).sum(1, dtype=F))[:, None]).astype(F)
    q = np.zeros(n, L.RAY_QUERY)
    q["origin"], q["direction"] = o, d
    q["distance"] = rng.choice([F(1e9), F(5.0) * F(sc.voxel_extent)], n)
    return q


def box_tests(sc, q, can_start, oriented):
    """(hit, t) of every ray against every voxel."""
    e = F(sc.voxel_extent)
    c = ((sc.aabbs["minimum"] + sc.aabbs["maximum"]) * F(0.5))[None]
    r = e * F(0.5)
    ir = F(1.0) / r
    d = q["direction"][:, None].astype(F)
    o = q["origin"][:, None].astype(F) - c
    with np.errstate(all="ignore"):
        w = np.where((np.abs(o) * ir).max(-1, keepdims=True) < 1, F(-1), F(1)) if can_start else F(1)
        sgn = -np.sign(d)
        dp = r * w * sgn - o
        dp = dp / d if oriented else dp * np.where(d == 0, F(1e12), F(1.0) / d)
        ok = []
        for a in range(3):
            b, g = (a + 1) % 3, (a + 2) % 3
            ok.append((dp[..., a] >= 0) & (np.abs(o[..., b] + d[..., b] * dp[..., a]) < r) &
                      (np.abs(o[..., g] + d[..., g] * dp[..., a]) < r))
    t = np.full(dp.shape[:2], F(-1))
    hit = np.zeros(dp.shape[:2], bool)
    done = np.zeros(dp.shape[:2], bool)
    for a in range(3):
        use = ok[a] & ~done
        done |= ok[a]
        s = np.broadcast_to(sgn[..., a] != 0, use.shape)
        hit |= use & s
        t = np.where(use & s, dp[..., a], t)
    return hit, t


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["one", "row_x", "row_y", "row_z", "negative", "grid", "edge5", "edge03"])
def test_walk_matches_brute_force(name):
    from cube_tracing.frame import SceneBuffers
    from test_gpu_traversal import gpu_queries
    sc = scene(name)
    sb = SceneBuffers(sc)
    # 257 rays: a partial warp and a partial block; 4000: many of each
    for n in (1, 257, 4000):
        q = ray_set(sc, n, seed=n)
        hit, t = box_tests(sc, q, True, True)
        t = np.where(hit & (t > 0) & (t <= q["distance"][:, None]), t, F(np.inf))
        best = t.argmin(1)  # the lowest primitive on ties
        tb = t[np.arange(n), best]
        got = gpu_queries(sb.accel, q, True)
        found = np.isfinite(tb)
        assert np.array_equal(got["instance_id"] == 0, found)
        assert np.array_equal(got["primitive_id"][found], best[found])
        assert np.array_equal(got["t"][found], tb[found])
        # visibility, every second ray with a target voxel it may reach
        rng = np.random.default_rng(n)
        q["flags"] = (np.arange(n) % 2) * L.QUERY_CHECK_TARGET
        q["target_primitive"] = np.where(rng.random(n) < 0.5, np.where(found, best, 0), rng.integers(0, sc.voxel_count, n))
        hit, t = box_tests(sc, q, False, False)
        t = np.where(hit & (t >= 0) & (t <= q["distance"][:, None]), t, F(np.inf))
        ids = np.arange(sc.voxel_count)[None]
        checks = (q["flags"] & L.QUERY_CHECK_TARGET) != 0
        target = np.where(checks, q["target_primitive"], -1)[:, None]
        key = np.where(checks, t[np.arange(n), q["target_primitive"]], F(np.inf))[:, None]
        blocks = np.isfinite(t) & (ids != target) & ((t < key) | ((t == key) & (ids < target)))
        blocks |= np.isfinite(t) & ~np.isfinite(key) & (ids != target)
        assert np.array_equal(gpu_queries(sb.accel, q, False), (~blocks.any(1)).astype(np.uint8))
